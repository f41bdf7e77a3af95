// SpMM kernel for the dense-B operand form on PAIRS of SMs (thread-block clusters of two CTAs, tcgen05 cta_group::2).
//
// A pair tile is 512 rows x BN columns: each CTA holds two row tiles of 128 (two accumulators) and HALF of every B stage (64 k x
// BN / 2 columns); one tcgen05.mma.sp.cta_group::2 multiplies 256 rows (128 from each CTA) with the BN columns assembled from both
// halves.  Per k-tile of 128 a CTA takes in 36 KiB of A and 32 KiB of B.  With one row tile a CTA (256 rows): 18 + 32 KiB.
//
// What bounds it: the tensor pipe inside a tile of 512 rows (8 MMAs x BN / 2 clocks a k-tile: 960 of 973 measured without loads, 991 with
// them, BN = 240); in a tile of 256 rows the intake (48 to 50 KiB for 480 clocks of MMAs, 490 to 600 with loads); and the stores of finished tiles,
// which leave in bursts and hold up the loads of the next tile.  4096 x 1024, N = 16384, [N,K] to [N,M], many calls at the clock that the power
// limit leaves: 512 x 240 tiles 76.7 us (after a pause, at 1965 MHz, 68.2), 256 x 240 80.3 (71.2); MMAs 29, floor 26.
// The last tile of a pair of 256 rows is drained by both epilogue groups, and no group waits for its slowest warp before it starts
// (2976 x 2040, N = 1368, [N,K], one wave: 15.3 -> 14.0 us).
//
// Cluster protocol (rank 0 = leader, rank 1 = peer); every load stays local to the CTA that issues it:
//   * both CTAs run their own A producer, B producers and epilogue on their own shared / tensor memory;
//   * the peer forwards "my A blocks of k-tile it landed" and "my half of stage j landed" to the leader with remote
//     mbarrier arrivals on the leader's own a_full / b_full barriers (which expect two arrivals there: the leader's
//     loads and the peer's message), so the leader's MMA issuer waits on one barrier per hand-off;
//   * only the leader issues tensor-core work: tcgen05.cp.cta_group::2 copies each CTA's metadata image into that
//     CTA's tensor memory, tcgen05.mma.sp.cta_group::2 reads A and B from both CTAs' shared memory.  Copies and MMAs come
//     from one elected thread, which executes them in order (see vnm_spmm.cu);
//   * the leader's tcgen05.commit.cta_group::2 arrives on the ring-free / accumulator-full barriers of BOTH CTAs, and the
//     peer's epilogue warps arrive remotely on the leader's accumulator-empty barrier.
// No copy with cluster multicast is used anywhere.  Every wait is bounded (status bit, drain, return), and the two CTAs
// meet at a cluster barrier before tensor memory is freed, so neither leaves while the other may still touch it.
#include "vnm_internal.h"

#include <type_traits>

namespace vnm {

namespace {

constexpr int RT = 2;            // row tiles (accumulators) per CTA; a pair tile has 2 * RT = 4 row tiles
constexpr int PART = 40;         // columns per epilogue part / TMA store (several destinations, BN = 240)
constexpr int KB_PER_STAGE = 2;                     // K=32 blocks per B stage: one 16 KiB TMA box (smaller boxes keep the copy engine less busy)
constexpr int STAGES_PER_KT = 4 / KB_PER_STAGE;
constexpr int B_CHUNK_BYTES = KB_PER_STAGE * 32 * 128;  // 64 rows x 64 columns
constexpr int B_STAGE_BYTES = 2 * B_CHUNK_BYTES;    // 16 KiB: two 64-column slices of which BN / 2 columns are used (or BN / 2 n-rows of 64 k)
constexpr int OUT_STAGE_BYTES = TILE_M * PART * 2;  // 128 rows x 40 fp16 columns, staging of one TMA store
constexpr int BAR_BYTES = 640;
// What depends on the row tiles per CTA.  The rings and the metadata sets advance one k-tile at a time; a k-tile is 68 KiB with
// two row tiles, 50 KiB with one.  Only results with several destinations pass through staging buffers.
template <int R, bool MULTI>
struct Plan {
    static constexpr int SA = R == 1 ? 4 : 3;                          // A ring: k-tiles (each R blocks)
    static constexpr int SB = SA * STAGES_PER_KT;                      // B ring: stages of 64 rows x 128 columns (this CTA's half of two K=32 blocks of the MMAs)
    static constexpr int A_STAGE_BYTES = R * AM_BLOCK_BYTES;
    static constexpr int A_RING_BYTES = SA * A_STAGE_BYTES;
    static constexpr int B_RING_BYTES = SB * B_STAGE_BYTES;
    static constexpr int OUT_RING_BYTES = MULTI ? RT * OUT_STAGE_BYTES : 0;   // one staging buffer per accumulator
    static constexpr int SMEM_BYTES = A_RING_BYTES + B_RING_BYTES + OUT_RING_BYTES + BAR_BYTES + 1024;
    static_assert(A_STAGE_BYTES % 1024 == 0 && B_STAGE_BYTES % 1024 == 0, "swizzled staging needs 1024-byte alignment");
    static_assert(SMEM_BYTES <= 227 * 1024, "shared memory per CTA");
    static_assert((2 * SA + 2 * SB + 4) * 8 + 16 <= BAR_BYTES, "barrier area too small");
};
// Four single-thread roles and two epilogue groups of four warps: 384 threads may use 168 registers each, which holds an
// accumulator row (120 packed words) without any re-allocation between warpgroups.  (With 512 threads and setmaxnreg the
// MMAs of this kernel issued at 180-240 clocks instead of 120: 1700 clocks a k-tile, against 1380.)
constexpr int NUM_THREADS = 384;
constexpr int EPI_WARP0 = 4;
constexpr int TMEM_COLS = 512;
// tensor-memory columns: accumulator 0 from 0, accumulator 1 from 256 (at most 240 columns each); metadata sets of four columns a
// row tile at 240..255 (and for a third set of two row tiles at 496)
__device__ __forceinline__ uint32_t acc_col(int rt) { return (uint32_t)rt * 256u; }
template <int R, int BN>
__device__ __forceinline__ uint32_t meta_col(int set)
{
    if (BN == 256) return 256u + 4u * (uint32_t)set;
    if (R == 1) return 240u + 4u * (uint32_t)set;
    return set == 2 ? 496u : 240u + 8u * (uint32_t)set;
}

// ---- cluster helpers ----
__device__ __forceinline__ uint32_t cluster_ctarank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// shared::cluster address of the same shared-memory location in CTA `rank` of this cluster
__device__ __forceinline__ uint32_t mapa_shared(uint32_t saddr, uint32_t rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr)
{
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void cluster_sync_all()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// ---- tcgen05, cta_group::2 forms ----
__device__ __forceinline__ void tmem_alloc2(uint32_t *smem_result, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish2() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc2(uint32_t taddr, uint32_t ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// arrives on the barrier at this shared-memory offset in both CTAs once every tcgen05 operation issued so far by this
// thread has completed (in both CTAs)
__device__ __forceinline__ void tc_commit2(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((uint16_t)3)
                 : "memory");
}
// each CTA's shared-memory image (same offset in both) -> that CTA's tensor memory, 128 lanes x 128 bits
__device__ __forceinline__ void tc_cp2_128x128b(uint32_t taddr, uint64_t sdesc)
{
    asm volatile("tcgen05.cp.cta_group::2.128x128b [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}
// D[256 x N] (+)= A_sparse[256 x 32] * B[32 x N]: rows 0-127 / A / D / metadata of the leader, rows 128-255 of the peer;
// B columns 0..N/2-1 from the leader's shared memory, N/2..N-1 from the peer's
__device__ __forceinline__ void tc_mma2_sp_f16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t meta_tmem, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.sp.cta_group::2.kind::f16 [%0], %1, %2, [%3], %4, {%6, %6, %6, %6, %6, %6, %6, %6}, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(meta_tmem), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
}

// Warp roles:
//   warp 0      A producer: one bulk copy per k-tile and row tile.
//   warps 1, 2  B producers, alternate stages: one TMA box each (64 k of this CTA's half of the columns).  One thread issues a
//               stage in about 420 clocks (wait, expect, box): alone it held tiles of one row tile at 850 clocks a k-tile,
//               against 480 of their MMAs; two of them: 35.1 -> 27.0 us at 1024 x 8192, N = 3072 ([N,K]).
//   warp 3      tensor-memory owner in both CTAs; leader: MMA issuer; peer: forwards "A blocks landed" and "B half landed"
//               to the leader.
//   warps 4..11 epilogue of this CTA's two accumulators.
template <int R, int BN, bool MULTI>
__global__ void __launch_bounds__(NUM_THREADS, 1) spmm_dense_b_pair_kernel(const __grid_constant__ CUtensorMap tmap_tile, const __grid_constant__ CUtensorMap tmap_tile2,
                                                                           const __grid_constant__ CUtensorMap tmap_out, const __grid_constant__ OutMaps more_out,
                                                                           const SpmmParams p)
{
    static_assert(R == 1 || R == RT, "row tiles per CTA");  // R = 1: pair tiles of 256 rows for problems with few row tiles
    constexpr bool ONE = BN == 256;                         // one accumulator: a tile's MMAs wait for the drain of the one before
    static_assert((BN <= 240 && BN % 16 == 0) || (ONE && R == 1 && !MULTI), "the tensor-memory column plan");
    static_assert(!MULTI || BN == 6 * PART, "parts of a tile that leaves through TMA stores");
    using P = Plan<R, MULTI>;
    constexpr int SA = P::SA, SB = P::SB, A_STAGE_BYTES = P::A_STAGE_BYTES, A_RING_BYTES = P::A_RING_BYTES;
    constexpr int B_RING_BYTES = P::B_RING_BYTES, OUT_RING_BYTES = P::OUT_RING_BYTES;
    constexpr int HALF_N = BN / 2;   // columns of a B stage held by each CTA of the pair
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t *a_ring = smem;
    uint8_t *b_ring = smem + A_RING_BYTES;
    uint8_t *out_ring = smem + A_RING_BYTES + B_RING_BYTES;
    uint64_t *a_full = reinterpret_cast<uint64_t *>(smem + A_RING_BYTES + B_RING_BYTES + OUT_RING_BYTES);
    uint64_t *b_full = a_full + SA;
    uint64_t *a_free = b_full + SB;   // the MMAs that read this slot have completed (arrives in both CTAs)
    uint64_t *b_free = a_free + SA;
    // accumulator hand-off, a barrier pair for each.  R = 2: both accumulators of a CTA belong to the same tile.  R = 1: a CTA has
    // one row tile, so its two accumulators alternate between consecutive tiles (ti & 1) and the epilogue of one tile runs
    // beside the MMAs of the next.
    uint64_t *acc_full_bar = b_free + SB;      // [2]
    uint64_t *acc_empty_bar = acc_full_bar + 2;  // [2]
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty_bar + 2);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t crank = cluster_ctarank();
    const bool leader_cta = crank == 0;
    const int pair = (int)blockIdx.x >> 1, npairs = (int)gridDim.x >> 1;
    // tiles of the pair: groups of 2 * R row tiles x column tiles, in the banded order of tile_coords()
    const int mquads = (p.mtiles + 2 * R - 1) / (2 * R);
    const int total_tiles = mquads * p.ntiles;
    const int my_tiles = (pair < total_tiles) ? (total_tiles - pair + npairs - 1) / npairs : 0;
    const int total_it = my_tiles * p.ktiles;

    if (threadIdx.x == 0) {
        // in the leader a slot is full once its own loads have landed AND the peer has reported the same for its half
        for (int s = 0; s < SA; s++) mbar_init(&a_full[s], leader_cta ? 2 : 1);
        for (int s = 0; s < SB; s++) mbar_init(&b_full[s], leader_cta ? 2 : 1);
        for (int s = 0; s < SA; s++) mbar_init(&a_free[s], 1);
        for (int s = 0; s < SB; s++) mbar_init(&b_free[s], 1);
        for (int a = 0; a < 2; a++) {
            mbar_init(&acc_full_bar[a], 1);
            mbar_init(&acc_empty_bar[a], ONE ? 2 * 8 : 2 * 4);  // the four warps of one epilogue group (of both) in both CTAs
        }
        *abort_flag = 0;
        fence_barrier_init();
    }
    grid_dependency_wait();
    if (warp == 3) {
        tmem_alloc2(tmem_slot, TMEM_COLS);
        tmem_relinquish2();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // both CTAs' barriers exist before anyone arrives on them remotely
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    grid_launch_dependents();
    // row tile of accumulator rt of this CTA in pair tile (mq, *)
    auto row_tile = [&](int mq, int rt) { return mq * 2 * R + (int)crank * R + rt; };

    if (warp == 0) {
        // ---------------- A producer ----------------
        if (elect_one()) {
            int it = 0;
            bool alive = true;
            for (int tile = pair; alive && tile < total_tiles; tile += npairs) {
                int mq, nt_unused;
                tile_coords(tile, mquads, p.ntiles, p.group_m, &mq, &nt_unused);
                for (int kt = 0; kt < p.ktiles; ++kt, ++it) {
                    const int s = it % SA;
                    if (!wait_quiet(&a_free[s], ((uint32_t)(it / SA) & 1u) ^ 1u, abort_flag, p.status, DEV_TIMEOUT_PRODUCER)) { alive = false; break; }
                    mbar_arrive_expect_tx(&a_full[s], R * AM_BLOCK_BYTES);
#pragma unroll
                    for (int rt = 0; rt < R; rt++) {
                        // a row tile past the end of the matrix re-reads the last one; its rows are never stored
                        const int mt = row_tile(mq, rt) < p.mtiles ? row_tile(mq, rt) : p.mtiles - 1;
                        bulk_g2s_hint(a_ring + s * A_STAGE_BYTES + rt * AM_BLOCK_BYTES, p.am + ((size_t)mt * p.ktiles + kt) * AM_BLOCK_BYTES, AM_BLOCK_BYTES,
                                      &a_full[s], p.hint_a);
                    }
                    if (p.l2_ahead > 0) {
                        // the same blocks of a later k-tile (of this tile, or of the next one of this pair) on their way into L2
                        int kp = kt + p.l2_ahead, mqp = mq;
                        bool ok = true;
                        if (kp >= p.ktiles) {
                            kp -= p.ktiles;
                            ok = kp < p.ktiles && tile + npairs < total_tiles;
                            if (ok) tile_coords(tile + npairs, mquads, p.ntiles, p.group_m, &mqp, &nt_unused);
                        }
                        if (ok) {
#pragma unroll
                            for (int rt = 0; rt < R; rt++) {
                                const int mt = row_tile(mqp, rt) < p.mtiles ? row_tile(mqp, rt) : p.mtiles - 1;
                                bulk_prefetch_l2(p.am + ((size_t)mt * p.ktiles + kp) * AM_BLOCK_BYTES, AM_BLOCK_BYTES);
                            }
                        }
                    }
                }
            }
            if (*abort_flag) {
                for (int k = it > SA ? it - SA : 0; k < it; ++k) drain_slot(&a_full[k % SA], (uint32_t)(k / SA) & 1u, p.status);
            }
        }
        __syncwarp();
    } else if (warp == 1 || warp == 2) {
        // ---------------- B producer: this CTA's half of every stage ----------------
        if (elect_one()) {
            tma_prefetch_desc(&tmap_tile);
            tma_prefetch_desc(&tmap_tile2);
            const int per_tile = STAGES_PER_KT * p.ktiles;
            const int half = warp - 1;   // stages of this parity
            int j = half, s = half;
            uint32_t ph = 1;
            bool alive = true;
            for (int tile = pair; alive && tile < total_tiles; tile += npairs) {
                int mq_unused, nt;
                tile_coords(tile, mquads, p.ntiles, p.group_m, &mq_unused, &nt);
                const int n0 = nt * BN + (int)crank * HALF_N;  // first column of this CTA's half
                const bool wide = p.b_wide_ok && n0 + 128 <= p.N;
                for (int jl = half; jl < per_tile; jl += 2, j += 2) {
                    if (!wait_quiet(&b_free[s], ph, abort_flag, p.status, DEV_TIMEOUT_PRODUCER)) { alive = false; break; }
                    uint8_t *dst = b_ring + s * B_STAGE_BYTES;
                    if (p.gather_mode == GATHER_NONE) {  // ablation: no loads of B at all (timing floor; results are meaningless)
                        mbar_arrive(&b_full[s]);
                    } else {
                        // 64 rows x 128 columns (the MMAs read the first BN / 2), or BN / 2 rows (n) x 64 k
                        mbar_arrive_expect_tx(&b_full[s], p.b_nk ? HALF_N * 128 : B_STAGE_BYTES);
                        if (p.b_nk) {
                            tma_load_2d_hint(dst, &tmap_tile, jl * 64, n0, &b_full[s], p.hint_b);  // 128-byte swizzle
                        } else if (wide) {
                            tma_load_4d_hint(dst, &tmap_tile, 0, jl * 64, 0, n0 / 8, &b_full[s], p.hint_b);  // {64 columns, 64 rows, 2 slices} from column n0
                        } else {  // ragged right edge: two boxes that clip (and zero-fill) at N
                            for (int c = 0; c < 2; c++) tma_load_2d_hint(dst + c * B_CHUNK_BYTES, &tmap_tile2, n0 + c * 64, jl * 64, &b_full[s], p.hint_b);
                        }
                        if (p.l2_ahead > 0) {
                            // the same box of a later stage, on its way into L2
                            int jlp = jl + STAGES_PER_KT * p.l2_ahead, n0p = n0;
                            bool ok = true;
                            if (jlp >= per_tile) {
                                jlp -= per_tile;
                                ok = jlp < per_tile && tile + npairs < total_tiles;
                                if (ok) {
                                    int ntp;
                                    tile_coords(tile + npairs, mquads, p.ntiles, p.group_m, &mq_unused, &ntp);
                                    n0p = ntp * BN + (int)crank * HALF_N;
                                }
                            }
                            if (ok) {
                                if (p.b_nk) tma_prefetch_2d(&tmap_tile, jlp * 64, n0p);
                                else if (p.b_wide_ok && n0p + 128 <= p.N) tma_prefetch_4d(&tmap_tile, 0, jlp * 64, 0, n0p / 8);
                                else for (int c = 0; c < 2; c++) tma_prefetch_2d(&tmap_tile2, n0p + c * 64, jlp * 64);
                            }
                        }
                    }
                    if ((s += 2) >= SB) { s = half; ph ^= 1; }
                }
            }
            if (*abort_flag && p.gather_mode != GATHER_NONE) {
                for (int k = j > SB ? j - SB : half; k < j; k += 2) drain_slot(&b_full[k % SB], (uint32_t)(k / SB) & 1u, p.status);
            }
        }
        __syncwarp();
    } else if (warp == 3) {
        if (!leader_cta && elect_one()) {
            // ---------------- peer: forward "A blocks landed" and "my half of the stage landed" ----------------
            const uint32_t remote_a = mapa_shared(smem_u32(a_full), 0), remote_b = mapa_shared(smem_u32(b_full), 0);
            int sa = 0;
            uint32_t ph = 0;
            bool alive = true;
            for (int it = 0; alive && it < total_it; ++it) {
                if (!wait_one(&a_full[sa], ph, abort_flag, p.status, DEV_TIMEOUT_MMA)) break;
                mbar_arrive_cluster(remote_a + (uint32_t)sa * 8u);
#pragma unroll
                for (int st = 0; st < STAGES_PER_KT; st++) {
                    const int sb = STAGES_PER_KT * sa + st;
                    if (!wait_one(&b_full[sb], ph, abort_flag, p.status, DEV_TIMEOUT_MMA)) { alive = false; break; }
                    mbar_arrive_cluster(remote_b + (uint32_t)sb * 8u);
                }
                if (++sa == SA) { sa = 0; ph ^= 1; }
            }
        }
        if (leader_cta && elect_one()) {
            // ---------------- MMA issuer (leader) ----------------
            const bool b_nk = p.b_nk != 0;
            const uint32_t idesc0 = make_idesc_f16(2 * TILE_M, BN, true, 0u, !b_nk);
            const uint64_t adesc0 = make_smem_desc(smem_u32(a_ring), 16, 1024, 2);
            const uint64_t mdesc0 = make_smem_desc(smem_u32(a_ring) + A_IMG_BYTES, 0, 128, 0);
            // this CTA's half of a stage: N-major (two 64-column slices of 64 rows x 128 bytes, 128-byte swizzle; a K=32 block is
            // 32 rows = 4096 bytes further) or K-major (BN / 2 n-rows of 128 bytes = 64 k, 128-byte swizzle,
            // 8-row groups 1024 bytes apart; a K=32 block is 64 bytes further inside the row)
            const uint64_t bdesc0 = b_nk ? make_smem_desc(smem_u32(b_ring), 16, 1024, 2) : make_smem_desc(smem_u32(b_ring), B_CHUNK_BYTES, 1024, 2);
            const uint32_t kb_step = b_nk ? 64u : 32u * 128u;  // bytes between the K=32 blocks of a stage
            int sa = 0;            // A slot and metadata set; the k-tile's B stages are slots STAGES_PER_KT * sa ...
            uint32_t ph = 0;       // phase of all of them
            int left = total_it;   // k-tiles, this one included
            bool alive = true;
            for (int ti = 0; alive && ti < my_tiles; ++ti) {
                // accumulator set: R = 2 both (phase ti), R = 1 set ti & 1 (phase ti / 2)
                const int aset = R == 1 && !ONE ? (ti & 1) : 0;
                const uint32_t aphase = R == 1 && !ONE ? (uint32_t)(ti >> 1) & 1u : (uint32_t)ti & 1u;
                for (int kt = 0; kt < p.ktiles; ++kt) {
                    if (kt == 0 && !wait_one(&acc_empty_bar[aset], aphase ^ 1u, abort_flag, p.status, DEV_TIMEOUT_MMA)) { alive = false; break; }
                    if (!wait_one(&a_full[sa], ph, abort_flag, p.status, DEV_TIMEOUT_MMA)) { alive = false; break; }  // both CTAs' blocks
                    tc_fence_after();
                    // A slot is reported free only where a later k-tile will fill it: the peer leaves once the last accumulator is full and
                    // stored, and an arrival that none of its threads waits for could come after that.
                    const bool refilled = left > SA;
                    const uint32_t mcol = tmem_base + meta_col<R, BN>(sa);
                    const uint32_t aoff = (uint32_t)(sa * A_STAGE_BYTES) >> 4;
#pragma unroll
                    for (int rt = 0; rt < R; rt++) tc_cp2_128x128b(mcol + rt * 4, mdesc0 + aoff + (uint32_t)((rt * AM_BLOCK_BYTES) >> 4));
                    // The k-tile's MMAs of one row tile, then those of the other: the first accumulator of a tile is full half a
                    // k-tile before the second one, and its next tile may begin while the second one is still being read
                    // (the hand-off of both at once kept the tensor pipe idle for 2600 clocks a tile).
#pragma unroll
                    for (int rt = 0; rt < R; rt++) {
                        if (R == 2 && rt == 1 && kt == 0) {
                            if (!wait_one(&acc_empty_bar[1], aphase ^ 1u, abort_flag, p.status, DEV_TIMEOUT_MMA)) { alive = false; break; }
                            tc_fence_after();
                        }
#pragma unroll
                        for (int st = 0; st < STAGES_PER_KT; st++) {
                            const int sb = STAGES_PER_KT * sa + st;
                            if (rt == 0) {
                                if (!wait_one(&b_full[sb], ph, abort_flag, p.status, DEV_TIMEOUT_MMA)) { alive = false; break; }  // both halves
                                tc_fence_after();
                            }
#pragma unroll
                            for (int k2 = 0; k2 < KB_PER_STAGE; k2++) {  // K=32 blocks of the stage
                                const int kb = st * KB_PER_STAGE + k2;
                                const uint32_t boff = ((uint32_t)sb * B_STAGE_BYTES + (uint32_t)k2 * kb_step) >> 4;
                                tc_mma2_sp_f16(tmem_base + acc_col(R == 1 ? aset : rt), adesc0 + aoff + (uint32_t)((rt * AM_BLOCK_BYTES + kb * 32) >> 4), bdesc0 + boff,
                                               mcol + rt * 4 + (uint32_t)(kb & ~1), idesc0 | (uint32_t)(kb & 1), (kt | kb) != 0 ? 1u : 0u);
                            }
                            if (rt == R - 1 && refilled) tc_commit2(&b_free[sb]);
                        }
                        if (!alive) break;
                        if (kt == p.ktiles - 1) tc_commit2(&acc_full_bar[R == 1 ? aset : rt]);
                    }
                    if (!alive) break;
                    if (refilled) tc_commit2(&a_free[sa]);
                    --left;
                    if (++sa == SA) { sa = 0; ph ^= 1; }
                }
            }
        }
        __syncwarp();
    } else {
        // ---------------- epilogue (both CTAs, own accumulators) ----------------
        const int q = warp & 3;
        const int i = q * 32 + lane;
        const int arow = mma_row_to_actual(i);
        const int grp = (warp - EPI_WARP0) >> 2;  // R = 2: the accumulator (row tile) this group drains; R = 1: the tiles ti with ti & 1 == grp
        int ti = 0;
        for (int tile = pair; tile < total_tiles; tile += npairs, ++ti) {
            // R = 1: this group's tiles, its half of every tile (ONE), or its half of this CTA's last tile, with which the other has nothing
            // left to do
            const bool shared = ONE || (R == 1 && !MULTI && ti == my_tiles - 1);
            if (R == 1 && !shared && (ti & 1) != grp) continue;
            const int aset = R == 2 ? grp : ONE ? 0 : ti & 1;
            int mq, nt;
            tile_coords(tile, mquads, p.ntiles, p.group_m, &mq, &nt);
            const int n0 = nt * BN;
            // with several destinations the four warps of a group leave the loop together (they meet at named barriers below)
            const bool got = wait_warp(&acc_full_bar[aset], R == 1 && !ONE ? (uint32_t)(ti >> 1) & 1u : (uint32_t)ti & 1u, abort_flag, p.status,
                                       DEV_TIMEOUT_EPILOGUE);
            if (MULTI ? !named_barrier_and(1 + grp, 128, got) : !got) break;
            if constexpr (MULTI && R == 2) {
                // the last tile is staged in the rings, which the MMAs of the other row tile read half a k-tile longer than those of the first
                if (ti == my_tiles - 1 && grp == 0 &&
                    !named_barrier_and(1 + grp, 128, wait_warp(&acc_full_bar[1], (uint32_t)ti & 1u, abort_flag, p.status, DEV_TIMEOUT_EPILOGUE))) break;
            }
            tc_fence_after();
            {
                const int rt = R == 1 ? 0 : grp;  // row tile of this CTA
                const int mt = row_tile(mq, rt);
                const uint32_t empty_leader = mapa_shared(smem_u32(&acc_empty_bar[aset]), 0);
                auto release = [&] {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(empty_leader);  // the leader's MMA issuer waits for both CTAs' epilogues
                };
                if constexpr (!MULTI) {
                    // straight from tensor memory; with two row tiles per CTA the next tile's MMAs wait for both accumulators, so
                    // they are read into registers whole before the first store
                    const uint32_t tacc = tmem_base + ((uint32_t)(q * 32) << 16) + acc_col(aset);
                    auto store = [&](auto width, auto hold, int first) {
                        constexpr int W = decltype(width)::value;
                        constexpr bool HOLD = decltype(hold)::value;
                        if (p.layout == 0) store_tile<W, HOLD>(TileStoreMN(tacc + (uint32_t)first, q, (int64_t)mt * TILE_M, n0 + first, p), release);
                        else store_tile<W, HOLD>(TileStoreNM(tacc + (uint32_t)first, q, (int64_t)mt * TILE_M, n0 + first, p), release);
                    };
                    using std::integral_constant;
                    if constexpr (ONE) {
                        store(integral_constant<int, 128>(), integral_constant<bool, false>(), grp * 128);
                    } else if (!shared) {
                        store(integral_constant<int, BN>(), integral_constant<bool, R == 2>(), 0);
                    } else if (grp == 0) {
                        store(integral_constant<int, 128>(), integral_constant<bool, false>(), 0);
                    } else {
                        store(integral_constant<int, BN - 128>(), integral_constant<bool, false>(), 128);
                    }
                } else {
                const int64_t row = (int64_t)mt * TILE_M + arow;
                const bool row_ok = mt < p.mtiles && row < p.M;
                const bool has_bias = p.layout == 1 && p.bias != nullptr;
                const __half bias = (has_bias && row_ok) ? p.bias[row] : __ushort_as_half((unsigned short)0);
                const bool leader = (warp == EPI_WARP0 + 4 * grp) && lane == 0;
                const uint32_t trow = tmem_base + ((uint32_t)(q * 32) << 16) + acc_col(grp);
                // 40 accumulator columns of this thread's row -> 20 registers of packed halves
                auto drain = [&](int part, uint32_t *pk) {
                    uint32_t v0[32], v1[8];
                    tc_ld_32x32b_x32(trow + (uint32_t)(part * PART), v0);
                    tc_ld_32x32b_x8(trow + (uint32_t)(part * PART) + 32u, v1);
                    tc_wait_ld();
#pragma unroll
                    for (int jj = 0; jj < 16; jj++) {
                        __half2 h0 = __floats2half2_rn(__uint_as_float(v0[2 * jj]), __uint_as_float(v0[2 * jj + 1]));
                        pk[jj] = *reinterpret_cast<uint32_t *>(&h0);
                    }
#pragma unroll
                    for (int jj = 0; jj < 4; jj++) {
                        __half2 h1 = __floats2half2_rn(__uint_as_float(v1[2 * jj]), __uint_as_float(v1[2 * jj + 1]));
                        pk[16 + jj] = *reinterpret_cast<uint32_t *>(&h1);
                    }
                };
                // Several destinations: one part -> staging buffer -> one TMA store for each (which clips at M and N).  In the CTA's last tile nothing hides the
                // stores behind later MMAs any more, and the operand rings are idle (every load has landed and every MMA that
                // read them has completed, or this CTA's accumulators would not be full): each part then gets a buffer of its
                // own inside the rings, so no part waits for the previous store to release the staging buffer (final epilogue 9.6k ->
                // 6.5k clocks; laying the six parts side by side and storing the 128 x 240 image at once measured slower, 8.1k).
                const bool last_tile = ti == my_tiles - 1;
                static_assert(RT * (BN / PART) * OUT_STAGE_BYTES <= A_RING_BYTES + B_RING_BYTES, "the last tile's staging does not fit into the rings");
                auto store_part = [&](int part, const uint32_t *pk) {
                    const bool in_range = mt < p.mtiles && n0 + part * PART < p.N;
                    uint8_t *stg = last_tile ? a_ring + (size_t)(grp * (BN / PART) + part) * OUT_STAGE_BYTES : out_ring + grp * OUT_STAGE_BYTES;
                    if (!last_tile) {
                        if (leader) bulk_wait_group_read0();  // the previous store has finished reading the staging buffer
                        named_barrier_sync(1 + grp, 128);
                    }
                    if (p.layout == 0) {
#pragma unroll
                        for (int c = 0; c < PART / 8; c++)
                            *reinterpret_cast<uint4 *>(stg + arow * (PART * 2) + c * 16) = make_uint4(pk[4 * c], pk[4 * c + 1], pk[4 * c + 2], pk[4 * c + 3]);
                    } else {
                        __half *col = reinterpret_cast<__half *>(stg) + arow;
#pragma unroll
                        for (int jj = 0; jj < PART / 2; jj++) {
                            uint32_t pw = pk[jj];
                            __half2 h = *reinterpret_cast<__half2 *>(&pw);
                            __half lo = __low2half(h), hi = __high2half(h);
                            if (has_bias) { lo = __hadd(lo, bias); hi = __hadd(hi, bias); }
                            col[(2 * jj) * TILE_M] = lo;
                            col[(2 * jj + 1) * TILE_M] = hi;
                        }
                    }
                    fence_proxy_async();
                    named_barrier_sync(1 + grp, 128);
                    if (leader && in_range) {
                        const int cx = p.layout == 0 ? n0 + part * PART : mt * TILE_M, cy = p.layout == 0 ? mt * TILE_M : n0 + part * PART;
                        tma_store_2d(&tmap_out, stg, cx, cy);
                        // further destinations of the same tile (the same rows of the peers' result buffers), one group with the first
                        for (int d = 1; d < p.n_out; d++) tma_store_2d(&more_out.m[d - 1], stg, cx, cy);
                        bulk_commit_group();
                    }
                };
                constexpr int NPARTS = BN / PART, HELD = R == 2 ? 5 : 1;  // R = 1: the next tile has the other accumulator
#pragma unroll
                for (int part = 0; part < NPARTS - HELD; part++) {
                    uint32_t pk[PART / 2];
                    drain(part, pk);
                    store_part(part, pk);
                }
                uint32_t held[HELD * (PART / 2)];
#pragma unroll
                for (int h = 0; h < HELD; h++) drain(NPARTS - HELD + h, held + h * (PART / 2));
                release();
#pragma unroll
                for (int h = 0; h < HELD; h++) store_part(NPARTS - HELD + h, held + h * (PART / 2));
                }
            }
        }
    }

    if (MULTI && warp >= EPI_WARP0 && ((warp - EPI_WARP0) & 3) == 0 && lane == 0) bulk_wait_group_read0();  // this thread's TMA stores have read shared memory (their global writes complete with the grid)
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // the peer's shared and tensor memory stay alive until the leader's last MMA and commit are done: the epilogues have seen the last commit arrive
    if (warp == 3) {
        tc_fence_after();
        tmem_dealloc2(tmem_base, TMEM_COLS);
    }
}

int g_pair_clusters = 0;  // co-resident clusters of two CTAs on this device (0 = not queried yet)

}  // namespace

#define VNM_PAIR_INSTANCES(X) X(1, 256, false) X(1, 192, false) X(1, 224, false) X(1, 240, false) X(1, 240, true) X(2, 192, false) X(2, 224, false) X(2, 240, false) X(2, 240, true)

cudaError_t spmm_dense_b_pair_init()
{
    cudaError_t e;
#define VNM_PAIR_ATTR(R, BN, MULTI) \
    if ((e = cudaFuncSetAttribute(spmm_dense_b_pair_kernel<R, BN, MULTI>, cudaFuncAttributeMaxDynamicSharedMemorySize, Plan<R, MULTI>::SMEM_BYTES)) != cudaSuccess) return e;
    VNM_PAIR_INSTANCES(VNM_PAIR_ATTR)
#undef VNM_PAIR_ATTR
    int dev = 0, sms = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)(sms & ~1), 1, 1);
    lc.blockDim = dim3(NUM_THREADS, 1, 1);
    lc.dynamicSmemBytes = Plan<1, false>::SMEM_BYTES;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    lc.attrs = attr;
    lc.numAttrs = 1;
    int clusters = 0;
    e = cudaOccupancyMaxActiveClusters(&clusters, spmm_dense_b_pair_kernel<1, 240, false>, &lc);
    if (e != cudaSuccess) { (void)cudaGetLastError(); clusters = 0; }
    g_pair_clusters = clusters;
    return cudaSuccess;
}

// Pair tiles have 512 rows (two row tiles per CTA) or 256 (one row tile per CTA) and 256, 240, 224 or 192 columns.  The tall form reads every
// B stage once per 512 rows, but its accumulators are drained between tiles and it needs twice the rows for a full wave; row tiles that
// do not divide evenly are padded (computed, never stored).  256 columns leave tensor memory for one accumulator only: the MMAs wait
// while it is drained, by both epilogue groups.  A [K,N] operand never takes 240 columns: the peer's half, 240 bytes further, starts
// inside a 32-byte sector (0.65 us a k-tile instead of 0.48); 256 are aligned, and one wave of such tiles is what it wants most often:
// 1024 x 4096, N = 4096 26.1 us as 512 x 192 (44 tiles for 74 pairs), 19.8 as 256 x 256; 8192 x 2048, N = 1024 25.2, 18.7; 4096 x 4096, N =
// 4096 70.9, 64.2.  [N,K]: 256 x 240 or 256 where tiles are few, else 512 x 240.
// The cost of a call, us: a start, and per wave a k-tile's time and a drain, with waves between the whole number that the last tile makes
// and the fraction that the SMs' power and memory see.  Fitted to steady calls on inputs that change, 22 shapes from 512 to 49152 rows, 512
// to 12288 k and 512 to 16384 columns, both layouts, all seven tiles (ratio to the measured time 0.7 to 1.25); the tile chosen takes
// 1.007 of the fastest one's time on average, 1.16 at most (2048 x 8192, N = 1000, whose rows of 2000 bytes are not aligned to sectors).
float spmm_dense_b_pair_config(int M, int N, int K, int b_nk, int max_ctas, int force_rows, bool multi, SpmmConfig *cfg)
{
    if (g_pair_clusters <= 0) return -1.0f;
    const int mtiles = (M + TILE_M - 1) / TILE_M, ktiles = (K + 127) / 128;
    int clusters = g_pair_clusters;
    if (max_ctas > 0 && max_ctas / 2 < clusters) clusters = max_ctas / 2;
    if (clusters < 1) return -1.0f;
    static const int widths[4] = {256, 240, 224, 192};
    struct Cost { float start, kt, wave; };
    static const Cost cost[2][2][4] = {   // [row tiles - 1][b_nk][width], us
        {{{4.2f, 0.533f, 1.3f}, {6.0f, 0.692f, 0.95f}, {5.2f, 0.519f, 1.1f}, {5.45f, 0.506f, 0.85f}}, {{4.4f, 0.507f, 1.5f}, {4.5f, 0.474f, 1.25f}, {4.7f, 0.462f, 1.05f}, {4.95f, 0.429f, 0.9f}}},
        {{{0.0f, 0.0f, 0.0f}, {4.85f, 1.006f, 2.75f}, {4.65f, 0.847f, 3.0f}, {4.1f, 0.792f, 2.45f}}, {{0.0f, 0.0f, 0.0f}, {4.2f, 0.853f, 2.75f}, {4.9f, 0.808f, 2.95f}, {4.4f, 0.729f, 2.25f}}}};
    float best = 1e30f;
    for (int w = 0; w < 4; w++) {
        if (multi ? widths[w] != 6 * PART : !b_nk && widths[w] == 240) continue;
        const long long ntiles = (N + widths[w] - 1) / widths[w];
        for (int rt = 1; rt <= RT; rt++) {
            if (rt == RT && widths[w] == 256) continue;   // its accumulators would fill tensor memory
            if ((force_rows == 1 && rt == RT) || (force_rows == 2 && mtiles > 2 && rt == 1)) continue;
            const long long tiles = (long long)((mtiles + 2 * rt - 1) / (2 * rt)) * ntiles;
            const float waves = 0.6f * (float)((tiles + clusters - 1) / clusters) + 0.4f * (float)tiles / clusters;
            const Cost &c = cost[rt - 1][b_nk != 0][w];
            const float us = c.start + waves * (ktiles * c.kt + c.wave);
            if (us < best) {
                best = us;
                cfg->bn = widths[w];
                cfg->nb = 2 * rt;  // row tiles per pair tile
                cfg->smem_bytes = rt == RT ? (multi ? Plan<2, true>::SMEM_BYTES : Plan<2, false>::SMEM_BYTES) : (multi ? Plan<1, true>::SMEM_BYTES : Plan<1, false>::SMEM_BYTES);
                cfg->grid = 2 * (int)(tiles < clusters ? tiles : clusters);
            }
        }
    }
    cfg->part = PART;
    cfg->stages = 2;
    cfg->threads = NUM_THREADS;
    return best;
}

cudaError_t launch_spmm_dense_b_pair(const SpmmConfig &cfg, const CUtensorMap &tmap_tile, const CUtensorMap &tmap_tile2, const CUtensorMap &tmap_out, const OutMaps &more_out,
                                     const SpmmParams &p, cudaStream_t stream)
{
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)cfg.grid, 1, 1);
    lc.blockDim = dim3(NUM_THREADS, 1, 1);
    lc.dynamicSmemBytes = (size_t)cfg.smem_bytes;
    lc.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    lc.attrs = attr;
    attr[1] = early_launch();
    lc.numAttrs = 2;
    const bool multi = p.n_out > 1;
#define VNM_PAIR_LAUNCH(R, BN, MULTI) \
    if (cfg.nb == 2 * R && cfg.bn == BN && multi == MULTI) return cudaLaunchKernelEx(&lc, spmm_dense_b_pair_kernel<R, BN, MULTI>, tmap_tile, tmap_tile2, tmap_out, more_out, p);
    VNM_PAIR_INSTANCES(VNM_PAIR_LAUNCH)
#undef VNM_PAIR_LAUNCH
    return cudaErrorInvalidValue;
}

}  // namespace vnm
