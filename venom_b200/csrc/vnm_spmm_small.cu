// SpMM kernel for few columns: C[M,N] = A * B for decoding steps and other products with too few large tiles to occupy the
// GPU.  Both operand forms: the V:N:M form (rows of B gathered, NB = 128/V blocks) and the dense-B form (B as [K,N] or [N,K]
// tiles shared by all blocks, NB = 1).
//
// Such products are bound by reading A once (a decoding step) or by latency (everything small), not by MMAs.  So a tile is
// 128 rows x BN = 16, 32, 64 or 128 columns, two CTAs share an SM (one loads while the other starts or stores), and
// when the row tiles do not fill the GPU a cluster of up to eight CTAs splits the k-tiles of one tile: the partial sums
// travel through distributed shared memory, each CTA adds up and stores its share of the columns, always in rank order, so
// results are the same on every call.
//
// One ring stage is a whole k-tile: the 18 KiB block of A (values and metadata, one bulk copy) and its rows of B.
// Warps: 0..7 B producers (gather4 loads dealt to all of them; plain tiles: warps 0 and 1 in turn), 8 A producer (with warp 10 in turn in the
// deep instances), 9 tensor-memory owner and MMA issuer, 12..15 epilogue.  Every wait is bounded.  One thread needs up to 420 clocks to issue
// a stage: 15.9 us a layer at 2048 x 8192, 128:2:8, 96 tokens with one issuing warp for B and A each, 13.8 with two.  Deep instances issue gathers
// from one elected lane (see vnm_spmm.cu): 18.8 -> 15.8 us at 2048 x 8192, 128:2:8, N = 96 in tiles of 128 columns, 10.7 -> 9.5 at 1024 x 4096, 64:2:8,
// N = 64; with two CTAs an SM it is bound by A and a gather4 a lane is as fast or faster (36864 x 12288, 128:2:16, 16 tokens 27.5, 27.8).
#include "vnm_internal.h"

#include <cmath>
#include <cstring>

namespace vnm {

namespace {

template <int BN, int NB, bool DEEP>
struct Small {
    static_assert(NB == 1 || NB == 2 || NB == 4, "128 rows hold 1, 2 or 4 vector blocks");
    static constexpr int RB = BN >= 64 ? 128 : 2 * BN;        // bytes of a row of B in one slice (its swizzle span)
    static constexpr int SWIZZLE = RB == 128 ? 2 : RB == 64 ? 4 : 6;   // descriptor code
    static constexpr int CH = (BN + 63) / 64;                 // 64-column slices
    static constexpr int B_CHUNK_BYTES = KT_ROWS * RB;        // one slice of a block: the k-tile's 128 rows
    static constexpr int B_BLOCK_BYTES = CH * B_CHUNK_BYTES;
    static constexpr int B_BYTES = NB * B_BLOCK_BYTES;
    static constexpr int STAGE_BYTES = AM_BLOCK_BYTES + B_BYTES;
    static constexpr int PW = 8;
    static constexpr int GATHERS = NB * KT_GROUPS * CH;       // per k-tile
    static constexpr int PER_WARP = GATHERS / PW;
    static_assert(PER_WARP <= 32 && GATHERS % PW == 0 && KT_GROUPS % (NB * KT_GROUPS / PW) == 0, "gathers are dealt to the producer warps, groups of one block");
    // Gathers: a lane issues one each, or (where one CTA has the SM, and the eight groups of a warp fit every lane's registers) one lane all of a warp's
    static constexpr bool BY_LANE = !DEEP || NB == 4;
    // Two CTAs share an SM and each has half of its shared memory for the ring; one that has its SM to itself (DEEP) has all of it.
    static constexpr int RING_BYTES = (DEEP ? 210 : 104) * 1024, MOST = DEEP ? 8 : 5;
    static constexpr int STAGES = RING_BYTES / STAGE_BYTES < 2 ? 2 : RING_BYTES / STAGE_BYTES > MOST ? MOST : RING_BYTES / STAGE_BYTES;
    static constexpr int RED_BYTES = (BN + 8) * TILE_M * 4;   // split over K: this CTA's columns from every rank (8: its share is rounded up); in the idle rings
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 256 + 1024;
    static_assert(SMEM_BYTES <= 227 * 1024 && (BN > 64 || RED_BYTES <= STAGES * STAGE_BYTES), "shared memory per CTA");
    static constexpr bool TWO_FIT = 2 * (SMEM_BYTES + 1024) <= 227 * 1024;
    static constexpr int CTAS = !DEEP && TWO_FIT ? 2 : 1;     // resident per SM
    static constexpr int A_WARP = PW, MMA_WARP = PW + 1, A_WARP2 = PW + 2, EPI_WARP0 = 12;
    static constexpr int A_WARPS = DEEP ? 2 : 1;              // warps that load A
    static constexpr int NUM_THREADS = 16 * 32;
    static constexpr int META_COL = BN < 64 ? 64 : BN;        // the epilogue reads 64 columns at a time
    static constexpr int META_SETS = 4;
    static constexpr int TMEM_COLS = META_COL + 4 * META_SETS <= 128 ? 128 : 256;
};

__device__ __forceinline__ uint32_t cluster_ctarank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t mapa_shared(uint32_t saddr, uint32_t rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_cluster(uint32_t addr, uint32_t v) { asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }

template <int BN, int NB, bool DEEP>
__global__ void __launch_bounds__(Small<BN, NB, DEEP>::NUM_THREADS, 2)
    spmm_small_kernel(const __grid_constant__ CUtensorMap tmap_b, const SpmmParams p)
{
    using T = Small<BN, NB, DEEP>;
    static_assert(DEEP || T::TWO_FIT, "a CTA that has its SM to itself runs the deep instance");
    constexpr int S = T::STAGES;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t *b_ring = smem;                                   // swizzled tiles first: 1024-byte alignment
    uint8_t *a_ring = smem + S * T::B_BYTES;
    uint64_t *full = reinterpret_cast<uint64_t *>(a_ring + S * AM_BLOCK_BYTES);
    uint64_t *freed = full + S;
    uint64_t *acc_full = freed + S;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_full + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    int *fills = reinterpret_cast<int *>(tmem_slot + 2);      // k-tiles that a warp has issued loads of
    float *red = reinterpret_cast<float *>(smem);
    static_assert(T::B_BYTES % 1024 == 0 && (2 * S + 1) * 8 + 12 <= 256, "shared-memory plan");

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int split = p.split_k;
    const uint32_t rank = split > 1 ? cluster_ctarank() : 0u;
    const int tile = (int)blockIdx.x / split;
    const int mt = tile / p.ntiles, nt = tile - mt * p.ntiles;
    const int n0 = nt * BN;
    const int k0 = (int)((int64_t)p.ktiles * rank / split), k1 = (int)((int64_t)p.ktiles * (rank + 1) / split);
    const int mode = p.gather_mode;      // GATHER_TMA4, GATHER_CONTIG or GATHER_NONE
    const bool b_nk = p.b_nk != 0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(&full[s], 1 + (mode == GATHER_TMA4 ? T::PW : 1));   // the A producer and each warp that loads B
            mbar_init(&freed[s], 1);
        }
        mbar_init(acc_full, 1);
        *abort_flag = 0;
        *fills = 0;
        fence_barrier_init();
    }
    if (!p.early) grid_dependency_wait();
    if (warp == T::MMA_WARP) {
        tmem_alloc(tmem_slot, T::TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    grid_launch_dependents();

    if (warp < T::PW) {
        // ---------------- B producers ----------------
        if (p.early) grid_dependency_wait();   // B is still being written; A, barriers and tensor memory do not depend on it
        if (mode == GATHER_TMA4) {
            int kt = k0;
            if constexpr (T::BY_LANE) {
                const int q = warp * T::PER_WARP + lane;
                const bool on = lane < T::PER_WARP;
                const int gc = q % T::CH, gg = (q / T::CH) % KT_GROUPS, gb = on ? q / (T::CH * KT_GROUPS) : 0;
                const int4 *rows = p.rows + ((size_t)(mt * NB + gb) * p.ktiles) * KT_GROUPS + gg;
                if (lane == 0) tma_prefetch_desc(&tmap_b);
                int4 r = make_int4(0, 0, 0, 0);
                if (on && k0 < k1) r = __ldg(rows + (size_t)k0 * KT_GROUPS);
                int s = 0;
                uint32_t ph = 1;
                for (; kt < k1; ++kt) {
                    const int4 cur = r;
                    if (on && kt + 1 < k1) r = __ldg(rows + (size_t)(kt + 1) * KT_GROUPS);
                    if (!__all_sync(0xffffffffu, wait_quiet(&freed[s], ph, abort_flag, p.status, DEV_TIMEOUT_PRODUCER))) break;
                    if (lane == 0) mbar_arrive_expect_tx(&full[s], T::PER_WARP * 4 * T::RB);
                    __syncwarp();
                    if (on) tma_gather4(b_ring + s * T::B_BYTES + gb * T::B_BLOCK_BYTES + gc * T::B_CHUNK_BYTES + gg * 4 * T::RB, &tmap_b, n0 + gc * 64, cur, &full[s]);
                    if (++s == S) { s = 0; ph ^= 1; }
                }
            } else {
                // this warp's groups of a k-tile are warp * G ..; group q is group q % KT_GROUPS of vector block q / KT_GROUPS
                constexpr int G = NB * KT_GROUPS / T::PW;
                const int mine = warp * G;
                const int4 *entry = p.rows + ((size_t)(mt * NB + mine / KT_GROUPS) * p.ktiles + k0) * KT_GROUPS + mine % KT_GROUPS;
                uint8_t *const first = b_ring + mine / KT_GROUPS * T::B_BLOCK_BYTES + mine % KT_GROUPS * 4 * T::RB;
                if (lane == 0) tma_prefetch_desc(&tmap_b);
                int s = 0;
                uint32_t ph = 1;
                for (; kt < k1; ++kt) {
                    int4 rows[G];                    // on their way while the warp waits for the slot
#pragma unroll
                    for (int g = 0; g < G; g++) rows[g] = __ldg(entry + g);
                    entry += KT_GROUPS;
                    if (!__all_sync(0xffffffffu, wait_quiet(&freed[s], ph, abort_flag, p.status, DEV_TIMEOUT_PRODUCER))) break;
                    uint8_t *dst = first + s * T::B_BYTES;
                    if (elect_one()) {
                        mbar_arrive_expect_tx(&full[s], T::PER_WARP * 4 * T::RB);
#pragma unroll
                        for (int g = 0; g < G; g++) {
#pragma unroll
                            for (int c = 0; c < T::CH; c++) tma_gather4(dst + c * T::B_CHUNK_BYTES + g * 4 * T::RB, &tmap_b, n0 + c * 64, rows[g], &full[s]);
                        }
                    }
                    if (++s == S) { s = 0; ph ^= 1; }
                }
            }
            if (lane == 0) atomicMax(fills, kt - k0);
        } else if (warp < 2 && elect_one()) {
            tma_prefetch_desc(&tmap_b);
            int s = warp;
            uint32_t ph = 1;
            int kt = k0 + warp;
            for (; kt < k1; kt += 2) {
                if (!wait_quiet(&freed[s], ph, abort_flag, p.status, DEV_TIMEOUT_PRODUCER)) break;
                uint8_t *st = b_ring + s * T::B_BYTES;
                if (mode == GATHER_NONE) {
                    mbar_arrive(&full[s]);
                } else if (b_nk) {           // two boxes of BN n-rows x 64 k (NB == 1)
                    mbar_arrive_expect_tx(&full[s], 2 * BN * 128);
                    for (int h = 0; h < 2; h++) tma_load_2d(st + h * BN * 128, &tmap_b, kt * 128 + h * 64, n0, &full[s]);
                } else {                     // 128 consecutive rows; for NB > 1 every block reads the same ones
                    mbar_arrive_expect_tx(&full[s], T::B_BYTES);
                    for (int b = 0; b < NB; b++)
                        for (int c = 0; c < T::CH; c++) tma_load_2d(st + b * T::B_BLOCK_BYTES + c * T::B_CHUNK_BYTES, &tmap_b, n0 + c * 64, kt * KT_ROWS, &full[s]);
                }
                if ((s += 2) >= S) { s -= S; ph ^= 1; }
            }
            atomicMax(fills, kt - k0 - 1);
        }
        __syncwarp();
    } else if (warp == T::A_WARP || (T::A_WARPS == 2 && warp == T::A_WARP2)) {
        // ---------------- A producers, alternate k-tiles ----------------
        if (elect_one()) {
            const uint8_t *src = p.am + (size_t)mt * p.ktiles * AM_BLOCK_BYTES;
            constexpr int step = T::A_WARPS;
            const int half = warp == T::A_WARP ? 0 : 1;
            int s = half;
            uint32_t ph = 1;
            int kt = k0 + half;
            for (; kt < k1; kt += step) {
                if (!wait_quiet(&freed[s], ph, abort_flag, p.status, DEV_TIMEOUT_PRODUCER)) break;
                mbar_arrive_expect_tx(&full[s], AM_BLOCK_BYTES);
                bulk_g2s(a_ring + s * AM_BLOCK_BYTES, src + (size_t)kt * AM_BLOCK_BYTES, AM_BLOCK_BYTES, &full[s]);
                if ((s += step) >= S) { s -= S; ph ^= 1; }
            }
            atomicMax(fills, kt - k0 - step + 1);
        }
        __syncwarp();
    } else if (warp == T::MMA_WARP) {
        // ---------------- MMA issuer (see vnm_spmm.cu: one elected lane copies metadata and issues the MMAs behind it) ----------------
        if (elect_one()) {
            const uint32_t idesc0 = make_idesc_f16(TILE_M, BN, true, 0u, !b_nk);
            const uint64_t adesc0 = make_smem_desc(smem_u32(a_ring), 16, 1024, 2);
            const uint64_t mdesc0 = make_smem_desc(smem_u32(a_ring) + A_IMG_BYTES, 0, 128, 0);
            // N-major: slices of 128 rows of RB bytes, a K=32 block is 32 rows further.  K-major: two boxes of BN rows of 128 bytes
            // (64 k), a K=32 block is 64 bytes further inside a row.
            const uint64_t bdesc0 = b_nk ? make_smem_desc(smem_u32(b_ring), 16, 1024, 2) : make_smem_desc(smem_u32(b_ring), T::B_CHUNK_BYTES, 8 * T::RB, T::SWIZZLE);
            int s = 0;
            uint32_t ph = 0;
            for (int kt = k0; kt < k1; ++kt) {
                if (!wait_one(&full[s], ph, abort_flag, p.status, DEV_TIMEOUT_MMA)) break;
                tc_fence_after();
                const uint32_t mcol = tmem_base + (uint32_t)(T::META_COL + ((kt - k0) % T::META_SETS) * 4);
                const uint32_t aoff = (uint32_t)(s * AM_BLOCK_BYTES) >> 4, boff = (uint32_t)(s * T::B_BYTES) >> 4;
                tc_cp_128x128b(mcol, mdesc0 + aoff);
#pragma unroll
                for (int kb = 0; kb < 4; kb++) {
                    const uint32_t koff = b_nk ? (uint32_t)((kb >> 1) * BN * 128 + (kb & 1) * 64) : (uint32_t)(kb * 32 * T::RB);
#pragma unroll
                    for (int b = 0; b < NB; b++) {
                        uint32_t mk[4] = {0u, 0u, 0u, 0u};  // bit set = output lane NOT written
                        if (NB == 2) {
                            mk[0] = mk[1] = (b == 0) ? 0u : 0xFFFFFFFFu;
                            mk[2] = mk[3] = (b == 0) ? 0xFFFFFFFFu : 0u;
                        } else if (NB == 4) {
                            mk[0] = (b == 0) ? 0u : 0xFFFFFFFFu;
                            mk[1] = (b == 1) ? 0u : 0xFFFFFFFFu;
                            mk[2] = (b == 2) ? 0u : 0xFFFFFFFFu;
                            mk[3] = (b == 3) ? 0u : 0xFFFFFFFFu;
                        }
                        tc_mma_sp_f16(tmem_base, adesc0 + aoff + (uint32_t)(kb * 32 >> 4), bdesc0 + boff + ((koff + (uint32_t)(b * T::B_BLOCK_BYTES)) >> 4),
                                      mcol + (uint32_t)(kb & ~1), idesc0 | (uint32_t)(kb & 1), (kt != k0 || kb != 0) ? 1u : 0u, mk[0], mk[1], mk[2], mk[3]);
                    }
                }
                tc_commit(&freed[s]);
                if (++s == S) { s = 0; ph ^= 1; }
            }
            tc_commit(acc_full);   // on an abort, too: nothing of this thread is in flight when the CTA leaves
        }
        __syncwarp();
    }

    if (split == 1) {
        if (warp >= T::EPI_WARP0) {
            const int q = warp & 3;
            if (wait_warp(acc_full, 0u, abort_flag, p.status, DEV_TIMEOUT_EPILOGUE) && *abort_flag == 0) {
                tc_fence_after();
                const uint32_t trow = tmem_base + ((uint32_t)(q * 32) << 16);
                if (p.layout == 0) store_tile<BN, false>(TileStoreMN(trow, q, (int64_t)mt * TILE_M, n0, p), [] {});
                else store_tile<BN, false>(TileStoreNM(trow, q, (int64_t)mt * TILE_M, n0, p), [] {});
            }
        }
    } else if (BN <= 64) {
        // ---------------- split over K: rank d adds up columns [d * share, (d + 1) * share) of all ranks ----------------
        // A CTA whose waits ran out still takes part in the barriers; its sums are meaningless and the status word says so.
        const int share = (BN + split - 1) / split;
        if (warp >= T::EPI_WARP0) {
            (void)wait_warp(acc_full, 0u, abort_flag, p.status, DEV_TIMEOUT_EPILOGUE);
            tc_fence_after();
        }
        cluster_arrive();
        cluster_wait();                  // every MMA of every rank is done: the rings are free
        if (warp >= T::EPI_WARP0) {
            const int q = warp & 3;
            const uint32_t red0 = smem_u32(red) + (uint32_t)mma_row_to_actual(q * 32 + lane) * 4u;
            for (int c0 = 0; c0 < BN; c0 += 8) {
                uint32_t v[8];
                tc_ld_32x32b_x8(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)c0, v);
                tc_wait_ld();
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const int n = c0 + i, d = n / share;
                    st_cluster(mapa_shared(red0, (uint32_t)d) + (uint32_t)(((int)rank * share + n - d * share) * TILE_M * 4), v[i]);
                }
            }
        }
        __syncwarp();
        cluster_arrive();
        cluster_wait();                  // all partial sums have arrived, and nobody writes here any more
        const int first = (int)rank * share, count = first + share <= BN ? share : (BN > first ? BN - first : 0);
        for (int e = threadIdx.x; e < count * (TILE_M / 2); e += T::NUM_THREADS) {
            const int n = e / (TILE_M / 2), r2 = (e - n * (TILE_M / 2)) * 2;      // two neighbouring rows
            float2 sum = make_float2(0.0f, 0.0f);
            for (int d = 0; d < split; d++) {
                const float2 x = *reinterpret_cast<const float2 *>(red + (d * share + n) * TILE_M + r2);
                sum.x += x.x;
                sum.y += x.y;
            }
            const int64_t row = (int64_t)mt * TILE_M + r2;
            const int col = n0 + first + n;
            if (row >= p.M || col >= p.N) continue;
            __half2 h = __floats2half2_rn(sum.x, sum.y);
            if (p.layout == 0) {
                p.out[row * p.ldo + col] = __low2half(h);
                p.out[(row + 1) * p.ldo + col] = __high2half(h);
            } else {
                if (p.bias) h = __hadd2(h, __halves2half2(p.bias[row], p.bias[row + 1]));
                __half *d = p.out + (int64_t)col * p.ldo + row;
                if ((p.ldo & 1) == 0 && ((uintptr_t)p.out & 3) == 0) {
                    *reinterpret_cast<__half2 *>(d) = h;
                } else {
                    d[0] = __low2half(h);
                    d[1] = __high2half(h);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0 && *abort_flag) drain_ring(full, S, *fills, p.status);
    if (warp == T::MMA_WARP) {
        tc_fence_after();
        tmem_dealloc(tmem_base, T::TMEM_COLS);
    }
}

int g_num_sms_small = 0;

// Self-test of the bounded waits: two threads wait, through the same wait_one as the product kernels and with the
// same limit, on a barrier that nothing ever signals.  The first to run out of time records its status bit and
// raises the abort flag; the other sees the flag and leaves.  The kernel then returns normally.
__global__ void wait_expiry_selftest_kernel(int *status)
{
    __shared__ uint64_t bar;
    __shared__ int abort_word;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        abort_word = 0;
        fence_barrier_init();
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) wait_one(&bar, 0u, &abort_word, status, DEV_TIMEOUT_EPILOGUE);
    __syncthreads();
}

// The deep instance is the only one of a tile whose ring never lets a second CTA on the SM (64 columns of four blocks).
template <int BN, int NB>
constexpr bool only_deep = !Small<BN, NB, false>::TWO_FIT;

template <int BN, int NB, bool DEEP>
cudaError_t init_instance()
{
    return cudaFuncSetAttribute(spmm_small_kernel<BN, NB, DEEP>, cudaFuncAttributeMaxDynamicSharedMemorySize, Small<BN, NB, DEEP>::SMEM_BYTES);
}
template <int BN, int NB>
cudaError_t init_one()
{
    if constexpr (!only_deep<BN, NB>) {
        const cudaError_t e = init_instance<BN, NB, false>();
        if (e != cudaSuccess) return e;
    }
    return init_instance<BN, NB, true>();
}

template <int BN, int NB, bool DEEP>
cudaError_t launch_instance(const SpmmConfig &cfg, const CUtensorMap &tmap_b, const SpmmParams &p, cudaStream_t stream)
{
    using T = Small<BN, NB, DEEP>;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)cfg.grid, 1, 1);
    lc.blockDim = dim3(T::NUM_THREADS, 1, 1);
    lc.dynamicSmemBytes = T::SMEM_BYTES;
    lc.stream = stream;
    cudaLaunchAttribute attr[2];
    lc.attrs = attr;
    lc.numAttrs = 0;
    if (p.split_k > 1) {
        attr[lc.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attr[lc.numAttrs].val.clusterDim.x = (unsigned)p.split_k;
        attr[lc.numAttrs].val.clusterDim.y = 1;
        attr[lc.numAttrs++].val.clusterDim.z = 1;
    }
    attr[lc.numAttrs++] = early_launch();
    return cudaLaunchKernelEx(&lc, spmm_small_kernel<BN, NB, DEEP>, tmap_b, p);
}
template <int BN, int NB>
cudaError_t launch_one(const SpmmConfig &cfg, const CUtensorMap &tmap_b, const SpmmParams &p, cudaStream_t stream)
{
    if constexpr (!only_deep<BN, NB>) {
        if (!cfg.deep) return launch_instance<BN, NB, false>(cfg, tmap_b, p, stream);
    }
    return launch_instance<BN, NB, true>(cfg, tmap_b, p, stream);
}

// What a grid of the deep instance, or of the one that shares an SM, takes.
template <int BN, int NB>
void fill(SpmmConfig *cfg, bool deep)
{
    using Deep = Small<BN, NB, true>;
    using Shared = Small<BN, NB, false>;
    cfg->deep = deep || only_deep<BN, NB>;
    cfg->smem_bytes = cfg->deep ? Deep::SMEM_BYTES : Shared::SMEM_BYTES;
    cfg->threads = Deep::NUM_THREADS;
    cfg->resident = cfg->deep ? Deep::CTAS : Shared::CTAS;
}

#define VNM_SMALL_DISPATCH(bn, nb, CALL)                                                                                  \
    ((nb) == 1 ? ((bn) == 16 ? CALL(16, 1) : (bn) == 32 ? CALL(32, 1) : (bn) == 64 ? CALL(64, 1) : CALL(128, 1))           \
     : (nb) == 2 ? ((bn) == 16 ? CALL(16, 2) : (bn) == 32 ? CALL(32, 2) : CALL(64, 2))                                       \
                 : ((bn) == 16 ? CALL(16, 4) : (bn) == 32 ? CALL(32, 4) : CALL(64, 4)))

}  // namespace

cudaError_t launch_wait_expiry_selftest(int *status, cudaStream_t stream)
{
    wait_expiry_selftest_kernel<<<1, 64, 0, stream>>>(status);
    return cudaGetLastError();
}

cudaError_t spmm_small_init()
{
    cudaError_t e;
    if ((e = init_one<16, 1>()) != cudaSuccess || (e = init_one<32, 1>()) != cudaSuccess || (e = init_one<64, 1>()) != cudaSuccess ||
        (e = init_one<128, 1>()) != cudaSuccess || (e = init_one<16, 2>()) != cudaSuccess || (e = init_one<32, 2>()) != cudaSuccess ||
        (e = init_one<64, 2>()) != cudaSuccess || (e = init_one<16, 4>()) != cudaSuccess || (e = init_one<32, 4>()) != cudaSuccess ||
        (e = init_one<64, 4>()) != cudaSuccess)
        return e;
    int dev = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    return cudaDeviceGetAttribute(&g_num_sms_small, cudaDevAttrMultiProcessorCount, dev);
}

// Tile width and split with the smallest estimated time (microseconds, returned).  A fit to calls replayed from a graph, 512 x 4096 .. 36864 x
// 12288, N = 8 .. 1024, all widths, splits 1, 2, 3, 4, 6 and 8: a fixed part for launch, set-up, first loads and epilogue; a k-tile's time, with the
// deep ring where each CTA has an SM to itself and eight k-tiles or more to fill it with (4096 x 4096, N = 256, 64-column tiles 12.3 us a layer with two
// CTAs' rings, 10.9 with the deep one; fewer k-tiles, or a cluster of such CTAs, gain nothing or lose: 8.2 -> 10.8 at 1024 x 4096, N = 64, split by 8);
// the exchange of a split; a second CTA on an SM costs its set-up and shares the port; clusters of more than four do not
// fill the last SMs of a GPC; and A cannot be read faster than HBM delivers it.  The choice takes 1.006 of the fastest one's time on average, 1.06 at most,
// over 42 shapes (the fit to older kernels took 1.06 and 1.34: 14.2 us split by 3 instead of 10.6 by 2 at 12288 x 12288, 128:2:16, N = 16, 7.1 split by 8
// instead of 5.5 by 4 at 1024 x 4096, 64:2:8, N = 64).  Operands of every row (m = 4 in gather form) in several waves, where each vector block of a tile reads the
// same rows of B again, take 1.23, 1.40 and 1.66 of that fit on average and up to 2.4 (1, 2 and 4 blocks, 113 sizes), which is added beyond SMALL_SPLIT_N columns.
// Up to SMALL_SPLIT_N columns that fit prices the kernel against others, but its choice among widths and splits took up to 1.75 of the fastest one's time (1.041
// on average over 352 problems of 1024 x 1024 to 36864 x 12288, 8 to 64 columns, V = 128, 64 and 32, every width and split, weights in L2 where they fit; 1.76 and 1.038 from HBM): a cluster's exchange costs
// more the wider the tile, clusters of three leave SMs idle, a row of 16 bytes is slow to load, and a ring that shares its SM takes in the weights of the call behind.  So
// the choice has a cost of its own, with which it takes 1.31 and 1.015 (1.32 and 1.022;  12288 x 4096, 128:2:8, N = 32, [K,N] 15.1 us as 32 columns split by 2, 8.5 unsplit; 2944 x 2048, N = 64
// 9.9 as 32 columns split by 3, 5.8 unsplit).  Only up to SMALL_SPLIT_N columns are k-tiles split: beyond, the order of summation stays that of the other kernels,
// so that results do not depend on how a caller cuts its columns.
float spmm_small_config(int mtiles, int ktiles, int N, int nb, bool gather, bool every_row, bool b_nk, SpmmConfig *cfg)
{
    const int sms = g_num_sms_small > 0 ? g_num_sms_small : 148;
    static const int widths[4] = {16, 32, 64, 128};
    static const float fixed[4] = {3.15f, 3.3f, 4.0f, 4.65f};
    static const float kt_time[2][2][4] = {{{0.165f, 0.17f, 0.25f, 0.43f}, {0.165f, 0.17f, 0.172f, 0.24f}},      // [gather][deep][width]
                                           {{0.285f, 0.29f, 0.34f, 0.5f}, {0.285f, 0.29f, 0.27f, 0.35f}}};
    const float a_bytes = (float)mtiles * ktiles * AM_BLOCK_BYTES;
    const bool few = N <= SMALL_SPLIT_N;
    float estimate = 1e30f, best = 1e30f;
    for (int w = 0; w < 4; w++) {
        const int bn = widths[w];
        if ((bn == 128 && nb > 1) || (bn > 16 && bn >= 2 * N)) continue;
        SpmmConfig shared, alone;
        memset(&shared, 0, sizeof(shared));
        memset(&alone, 0, sizeof(alone));
#define VNM_FILL(BN, NB) (fill<BN, NB>(&shared, false), fill<BN, NB>(&alone, true))
        VNM_SMALL_DISPATCH(bn, nb, VNM_FILL);
#undef VNM_FILL
        const int tiles = mtiles * ((N + bn - 1) / bn);
        for (int split = 1; split <= 8 && split <= ktiles; split++) {
            const int ctas = tiles * split, kts = (ktiles + split - 1) / split;
            const bool deep = split == 1 && kts >= 8 && ctas <= sms;
            const bool one_each = (float)ctas <= (split <= 4 ? 1.0f : 0.72f) * sms;
            const float fit = (split <= 2 ? 1.0f : 0.89f) * (float)(sms * shared.resident);       // CTAs at a time
            const float kt_us = kt_time[gather][deep][w] * (nb == 4 ? 2.1f : nb == 2 ? 1.38f : 1.0f);
            float t = fixed[w] + (nb == 4 ? 1.0f : nb == 2 ? 0.2f : 0.0f);
            if (split > 1) t += 0.25f + 0.016f * bn + 0.004f * (float)(ctas < sms ? ctas : sms);
            if (one_each) t += kts * kt_us * (1.0f + (gather ? 0.1f * ctas / sms : 0.0f));
            else t += ceilf((float)ctas / fit) * (kts * kt_us * (every_row && !few ? 1.45f + 0.36f * nb : 1.45f) + 2.0f);
            const float hbm = 3.5f + a_bytes / (gather && one_each ? 4.2e6f : 5.6e6f);
            t = (t > hbm ? t : hbm) + 0.05f * t;
            estimate = t < estimate ? t : estimate;
            auto take = [&](float cost, bool deep_ring) {
                if (cost >= best) return;
                best = cost;
                *cfg = deep_ring ? alone : shared;
                cfg->bn = bn;
                cfg->nb = nb;
                cfg->part = bn;
                cfg->stages = 1;
                cfg->split = split;
                cfg->grid = ctas;
            };
            if (!few) {
                take(t, deep);
                break;
            }
            const bool at_once = (float)ctas <= (split > 4 ? 0.72f : split == 3 ? 0.81f : 1.0f) * sms;
            for (int ring = deep ? 1 : 0; ring >= 0; ring--) {
                float kt = kt_time[gather][ring][w] * (nb == 4 ? 2.1f : nb == 2 ? 1.38f : 1.0f);
                if (nb == 4) kt *= (bn == 64 ? 0.7f : 1.0f) * (every_row ? 1.54f : 1.0f);
                if (ring && (gather || (N < 16 && !b_nk))) kt *= 1.15f;
                if (N < 16 && !b_nk) kt *= 1.0f + (gather ? 0.55f : 0.5f * nb);      // rows of 16 bytes
                float cost = fixed[w] + (nb == 4 ? 1.0f : nb == 2 ? 0.2f : 0.0f);
                if (split > 1) cost += (0.038f + 0.15f / split) * bn - 0.4f;
                if (at_once) cost += kts * kt * (1.0f + (gather ? 0.1f * ctas / sms : 0.0f));
                else cost += ceilf((float)ctas / fit) * (split > 1 ? kts * kt * 1.32f + 3.1f : kts * kt * 1.45f + 2.0f);
                const float a_time = 3.5f + a_bytes / (!gather || !at_once ? 5.6e6f : ring ? 4.0e6f : split > 1 ? 4.7e6f : 5.6e6f);
                take((cost > a_time ? cost : a_time) + 0.05f * cost, ring != 0);
            }
        }
    }
    return estimate;
}

// Tensor map of the dense operand for this kernel: rows of at most 64 columns, gathered four at a time or as boxes of 128
// consecutive rows, or (b_nk) boxes of bn n-rows x 64 k.
CUresult spmm_small_encode(EncodeTiledFn enc, CUtensorMap *map, const void *B, int64_t ldb, int K, int N, int b_nk, int gather_mode, int bn)
{
    cuuint32_t estr[2] = {1, 1};
    cuuint64_t strides[1] = {(cuuint64_t)ldb * 2};
    if (b_nk) {
        cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)N};
        cuuint32_t box[2] = {64, (cuuint32_t)bn};
        return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(B), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    }
    cuuint64_t dims[2] = {(cuuint64_t)N, (cuuint64_t)K};
    const cuuint32_t w = bn >= 64 ? 64u : (cuuint32_t)bn;
    cuuint32_t box[2] = {w, gather_mode == GATHER_TMA4 ? 1u : 128u};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(B), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               w == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : w == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
}

cudaError_t launch_spmm_small(const SpmmConfig &cfg, const CUtensorMap &tmap_b, const SpmmParams &p, cudaStream_t stream)
{
#define VNM_LAUNCH(BN, NB) launch_one<BN, NB>(cfg, tmap_b, p, stream)
    return VNM_SMALL_DISPATCH(cfg.bn, cfg.nb, VNM_LAUNCH);
#undef VNM_LAUNCH
}

}  // namespace vnm
