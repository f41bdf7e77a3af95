// V:N:M SpMM for sm_100a: C[M,N] = A_vnm[M,K] * B[K,N], fp16 in, fp32 accumulate in tensor memory.
//
// Persistent kernel: one CTA per SM walks over 128 x BN output tiles (in the banded order of tile_coords(): the CTAs
// that run together share a few column panels of B and a band of row tiles of A that stays in L2).  The 128 rows of a
// tile hold NB = 128/V vector blocks; each block has its own column-loc, hence its own gathered rows of B.
//
// Two shared-memory rings feed the tensor core:
//   A ring  SA stages of 18 KiB: the value image (128 rows x 64 compressed columns, K-major, 128-byte swizzle) and the
//           metadata image of one k-tile, one bulk copy each;
//   B ring  SB stages of 16 KiB: 32 gathered rows (8 groups, one K=32 block of the MMAs) for each of the NB blocks,
//           N-major, 128-byte swizzle.
// Warp roles:
//   warps 0..15   B producers in eight pairs; pair j % 8 fills stage j, 16 TMA gather4 loads a warp (four absolute row
//                 numbers per instruction, precomputed by the prepare step).  One elected lane issues them, with the row numbers of its
//                 groups in its registers: 42 clocks a gather4.  (With a gather4 a lane, the warp goes through its lanes at 109 clocks
//                 each when all sixteen are at it, and the slots of the ring were waiting for that: 128.4 us at 12288 x 12288, 128:2:16, N = 2048,
//                 [K,N] to [M,N], many calls, against 117.2; 4096 x 4096, 128:2:8, N = 16384 218 and 197; 12288 x 12288, 64:2:32, N = 2048 113 and 106.)
//                 At V = 32 a warp has 16 groups of one gather4 each, too many for every lane to hold: there each lane holds and issues one
//                 (105 us at 4096 x 4096, 32:2:32, N = 8192; four warps a stage with eight groups each 111).  The row numbers are asked for
//                 before the wait for the slot, which takes longer.  (vnm_set_producer_warps, an ablation, leaves a quarter or half of the
//                 pairs at work.)
//   warp 16       A producer (one lane).
//   warp 17       tensor-memory owner and MMA issuer.  It waits for the operands itself, copies a k-tile's metadata to
//                 tensor memory (tcgen05.cp) and issues the MMAs right behind it: copies and MMAs of one thread execute
//                 in order, so nothing has to come back between them.  (With the copies in another thread, announced
//                 through tcgen05.commit and a barrier, each k-tile paid for that round trip: 2100-2500 clocks a k-tile
//                 with the loads of B switched off, against four MMAs of 152.)  The whole warp runs the loop and one elected
//                 lane issues, so that descriptors stay in uniform registers.
//   warps 18, 19  idle (the epilogue starts at a multiple of four warps: tensor-memory lane quadrants)
//   last eight    epilogue, two groups of four warps.  V = 128: each group drains half of the columns of the one accumulator.  V = 64
//                 and 32: consecutive tiles alternate between two accumulators, one for each group.
// V = 128: tiles of 256 columns fill whole gathers (64 columns each).  Two accumulators and the metadata would leave room for 240, of
// whose fourth gather a quarter goes unused.  With one accumulator the MMAs stop while a tile is drained (2800 clocks from the last MMA to the
// next one: 440 until the epilogue sees it, the rest to read and store half of its columns and read the others), and the rings (2.25 k-tiles)
// take in what arrives meanwhile.  Holding all columns in registers first needs more of them than 832 threads have.
// What bounds a k-tile now: 640 clocks of MMAs, whose operands and the 82 KiB of loads share the port of shared memory (900 without the
// loads of B, 1130 with them on 18 SMs, 1340 on all).
// [K,N] to [M,N], us, many calls (in brackets after a pause, 1965 MHz), 240 columns and two accumulators against 256 and one, without cut tiles
// and with a gather4 a lane:
//   12288 x 12288, m = 16, N = 2048: 143.0 (128.2), 131.7 (121.1);  4096 x 4096, N = 16384, m = 8: 241.0 (213.1), 217.0 (192.7), m = 16: 141.5 (124.9),
//   128.5 (113.5);  4096 x 512, m = 16 (one k-tile), N = 16384: 48.6 (50.0), 43.1 (44.3);  49152 x 12288, m = 8, N = 32768: 16040 (13880), 15444 (13304).
// A tenth B stage in the place of the staging buffers: 0.5 to 1 % faster up to 0.2 ms, slower at the largest.  A fourth A stage or L2 prefetches
// of A six k-tiles ahead: no change, 1 to 2 % slower.
// For NB > 1 each MMA runs on all 128 rows of the value tile with the output lanes of the other blocks disabled.
// Every wait is bounded: on expiry the kernel records a status bit, drains and returns.
#include "vnm_internal.h"

namespace vnm {

namespace {

constexpr int BS_ROWS = 32;     // gathered rows per B stage and block: one K=32 block of the MMAs
constexpr int BS_GROUPS = 8;    // groups per B stage and block
constexpr int STAGES_PER_KT = KT_ROWS / BS_ROWS;

template <int BN, int NB>
struct Traits {
    static_assert(NB == 1 || NB == 2 || NB == 4, "128 rows hold 1, 2 or 4 vector blocks");
    static constexpr int CH = (BN + 63) / 64;                 // 64-column slices per block
    static constexpr int B_CHUNK_BYTES = BS_ROWS * 128;       // one slice: 32 rows x 128 B
    static constexpr int B_BLOCK_BYTES = CH * B_CHUNK_BYTES;
    static constexpr int B_STAGE_BYTES = NB * B_BLOCK_BYTES;
    static constexpr bool CAN_CUT = CH > 1;                   // the last tiles of a launch may be cut in two
    static constexpr int GATHERS = NB * BS_GROUPS * CH;       // gather4 instructions per B stage (always 32)
    // 256 columns: one accumulator, which the two epilogue groups drain half and half.  Fewer: two that alternate between tiles.
    static constexpr int ACCS = BN == 256 ? 1 : 2;
    static constexpr int SA = 3, SB = 9;
    static constexpr int H = 2;                  // producer warps that share a stage
    static constexpr int PW = 16;
    static constexpr int NG = PW / H;
    static constexpr int GROUPS = NB * BS_GROUPS / H;         // groups of a stage that a warp gathers, CH instructions each
    static constexpr bool BY_LANE = NB == 4;                  // sixteen groups: a lane holds the rows of each (else every lane those of all)
    static_assert(GATHERS == 32 && (!BY_LANE || (GROUPS <= 32 && CH == 1)), "a stage is dealt to the warps by groups");
    static constexpr int A_WARP = PW, MMA_WARP = PW + 1, EPI_WARP0 = PW + 4;
    static constexpr int NUM_WARPS = EPI_WARP0 + 8;
    static constexpr int NUM_THREADS = NUM_WARPS * 32;
    static constexpr int DRAIN = ACCS == 1 ? BN / 2 : BN;     // columns of a tile that an epilogue group drains
    static constexpr int PART = 32;                           // columns per part of the epilogue that stores through TMA
    static_assert(BN % 64 == 0 && DRAIN % 64 == 0, "whole slices and epilogue chunks, also of half a tile");
    static_assert(64 % (2 * PART) == 0, "parts are read two at a time");
    static constexpr int A_RING_BYTES = SA * AM_BLOCK_BYTES;
    static constexpr int B_RING_BYTES = SB * B_STAGE_BYTES;
    static constexpr int OUT_STAGE_BYTES = TILE_M * PART * 2;
    static constexpr int BAR_BYTES = 512;
    static constexpr int OUT_RING_BYTES = 2 * OUT_STAGE_BYTES;
    static constexpr int SMEM_BYTES = A_RING_BYTES + B_RING_BYTES + OUT_RING_BYTES + BAR_BYTES + 1024;  // + alignment slack
    static_assert(SMEM_BYTES <= 227 * 1024, "shared memory per CTA");
    static_assert((2 * SA + 2 * SB + 4) * 8 + 16 <= BAR_BYTES, "barrier area too small");
    static_assert(A_RING_BYTES % 1024 == 0 && B_STAGE_BYTES % 1024 == 0 && OUT_STAGE_BYTES % 1024 == 0, "swizzled tiles need aligned rings");
    // tensor memory: the accumulators, three alternating metadata sets of four columns behind them
    static constexpr int META_COL = ACCS * BN;
    static constexpr int META_SETS = 3;
    static constexpr int TMEM_COLS = META_COL + META_SETS * 4 > 256 ? 512 : 256;
};

template <int BN, int NB>
__global__ void __launch_bounds__(Traits<BN, NB>::NUM_THREADS, 1)
    spmm_kernel(const __grid_constant__ CUtensorMap tmap_rows, const __grid_constant__ CUtensorMap tmap_tile, const __grid_constant__ CUtensorMap tmap_out,
                const __grid_constant__ OutMaps more_out, const SpmmParams p, const int cut_from)
{
    using T = Traits<BN, NB>;
    constexpr int SA = T::SA, SB = T::SB;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t *a_ring = smem;
    uint8_t *b_ring = a_ring + T::A_RING_BYTES;
    uint8_t *out_ring = b_ring + T::B_RING_BYTES;
    uint64_t *a_full = reinterpret_cast<uint64_t *>(out_ring + T::OUT_RING_BYTES);
    uint64_t *a_free = a_full + SA;
    uint64_t *b_full = a_free + SA;
    uint64_t *b_free = b_full + SB;
    uint64_t *acc_full = b_free + SB;      // [2], one of which is used if there is one accumulator
    uint64_t *acc_empty = acc_full + 2;    // [2]
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + 2);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    int *b_fills = reinterpret_cast<int *>(tmem_slot + 2);   // B stages that a warp has issued loads of

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int gmode = p.gather_mode;
    const int my_tiles = (int)blockIdx.x < p.total_tiles ? (p.total_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < SA; s++) { mbar_init(&a_full[s], 1); mbar_init(&a_free[s], 1); }
        // each warp of a producer pair arrives once with its byte count (TMA modes) or once per lane behind its copies
        const uint32_t per_warp = gmode == GATHER_CPASYNC ? 32 + (p.hybrid_rows ? 1 : 0) : 1;
        for (int s = 0; s < SB; s++) { mbar_init(&b_full[s], T::H * per_warp); mbar_init(&b_free[s], 1); }
        for (int a = 0; a < 2; a++) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], T::ACCS == 1 ? 8 : 4); }
        *abort_flag = 0;
        *b_fills = 0;
        fence_barrier_init();
    }
    grid_dependency_wait();
    if (warp == T::MMA_WARP) {
        tmem_alloc(tmem_slot, T::TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    grid_launch_dependents();

    // tile of the launch -> row tile, first column, slices of 64 columns.  From `cut_from` on two numbers are the halves of one tile.
    auto locate_tile = [&](int tile, int *mt, int *n0, int *slices) {
        int nt, half = 0;
        *slices = T::CH;
        if (T::CAN_CUT && tile >= cut_from) {
            half = (tile - cut_from) & 1;
            tile = cut_from + ((tile - cut_from) >> 1);
            *slices = T::CH / 2;
        }
        tile_coords(tile, p.mtiles, p.ntiles, p.group_m, mt, &nt);
        *n0 = nt * BN + half * (BN / 2);
    };

    const int ng = T::NG * p.producer_warps / GATHER_PRODUCER_WARPS > 0 ? T::NG * p.producer_warps / GATHER_PRODUCER_WARPS : 1;   // groups of H warps at work
    if (warp < T::H * ng) {
        // ---------------- B producers: the groups of H warps take the stages in turn ----------------
        constexpr int G = T::GROUPS, HELD = T::BY_LANE ? 1 : G;
        const int part = warp % T::H, first = warp / T::H;
        const int per_tile = STAGES_PER_KT * p.ktiles;
        // this warp's groups of a stage are part * G ..; group q is group q % BS_GROUPS of vector block q / BS_GROUPS
        const int mine = part * G + (T::BY_LANE ? lane % G : 0);
        constexpr int BOXES = NB * T::CH;             // plain tiles: boxes per stage, a lane each
        static_assert(BOXES % T::H == 0, "boxes are dealt to the warps");
        const bool box_on = lane < BOXES / T::H;
        const int bc = (part * (BOXES / T::H) + lane) % T::CH, bb = box_on ? (part * (BOXES / T::H) + lane) / T::CH : 0;
        if (lane == 0) { tma_prefetch_desc(&tmap_rows); tma_prefetch_desc(&tmap_tile); }
        int tile_i = first / per_tile, jl = first - tile_i * per_tile, s = first;
        static_assert(T::NG <= SB, "a group's first stage has its own slot");
        uint32_t parity = 1;
        int n0 = 0, slices = T::CH;
        const int4 *entry = nullptr;                  // the row numbers of group `mine` in stage jl
        auto locate = [&] {
            int mt;
            locate_tile((int)blockIdx.x + tile_i * (int)gridDim.x, &mt, &n0, &slices);
            entry = p.rows + ((size_t)(mt * NB + mine / BS_GROUPS) * p.ktiles) * KT_GROUPS + (size_t)jl * BS_GROUPS + mine % BS_GROUPS;
        };
        if (tile_i < my_tiles) locate();
        int4 ahead = make_int4(0, 0, 0, 0);           // BY_LANE: asked for a stage earlier (5184 x 2176, 32:2:32, N = 4320 66.5 -> 61.5 us; elsewhere no change)
        if (T::BY_LANE && tile_i < my_tiles && (gmode == GATHER_TMA4 || gmode == GATHER_CPASYNC)) ahead = __ldg(entry);
        int issued = 0;
        while (tile_i < my_tiles) {
            int4 rows[HELD];                          // on their way while the warp waits for the slot
            if (gmode == GATHER_TMA4 || gmode == GATHER_CPASYNC) {
#pragma unroll
                for (int g = 0; g < HELD; g++) rows[g] = T::BY_LANE ? ahead : __ldg(entry + g);   // one block's
            }
            const int n = n0, cols = slices, k_row = jl * BS_ROWS;
            uint8_t *st = b_ring + s * T::B_STAGE_BYTES;
            uint64_t *full = &b_full[s], *free = &b_free[s];
            const uint32_t cur_parity = parity;
            jl += ng;
            s += ng;
            entry += ng * BS_GROUPS;
            if (s >= SB) { s -= SB; parity ^= 1; }
            if (jl >= per_tile) {
                do { jl -= per_tile; ++tile_i; } while (jl >= per_tile);
                if (tile_i < my_tiles) locate();
            }
            if (T::BY_LANE && tile_i < my_tiles && (gmode == GATHER_TMA4 || gmode == GATHER_CPASYNC)) ahead = __ldg(entry);
            if (!__all_sync(0xffffffffu, wait_quiet(free, cur_parity, abort_flag, p.status, DEV_TIMEOUT_PRODUCER))) break;
            auto slot = [&](int q) { return st + q / BS_GROUPS * T::B_BLOCK_BYTES + q % BS_GROUPS * 512; };   // of a group, first slice
            if (gmode == GATHER_TMA4) {
                if constexpr (T::BY_LANE) {
                    if (lane == 0) mbar_arrive_expect_tx(full, G * 512);
                    __syncwarp();
                    if (lane < G) tma_gather4(slot(mine), &tmap_rows, n, rows[0], full);
                } else if (elect_one()) {
                    mbar_arrive_expect_tx(full, G * 512 * cols);
                    uint8_t *dst = slot(mine);
#pragma unroll
                    for (int g = 0; g < G; g++) {
#pragma unroll
                        for (int c = 0; c < T::CH; c++)
                            if (c < T::CH / 2 || cols == T::CH) tma_gather4(dst + c * T::B_CHUNK_BYTES + g * 512, &tmap_rows, n + c * 64, rows[g], full);
                    }
                }
            } else if (gmode == GATHER_CONTIG) {   // 32 consecutive rows (m == 4: all of them are selected)
                if (lane == 0) mbar_arrive_expect_tx(full, T::B_STAGE_BYTES / T::H);
                __syncwarp();
                if (box_on) tma_load_2d(st + bb * T::B_BLOCK_BYTES + bc * T::B_CHUNK_BYTES, &tmap_tile, n + bc * 64, k_row, full);
            } else if (gmode == GATHER_NONE) {     // ablation: no loads of B (timing floor; results are meaningless)
                if (lane == 0) mbar_arrive(full);
            } else {
                // ablation: per-thread 16-byte asynchronous copies driven by the row table, optionally beside gather4 loads of
                // the first `by_tma` groups of every block
                const int by_tma = p.hybrid_rows / 8;
                if (by_tma > 0) {
                    int here = 0;
                    for (int g = 0; g < G; g++) here += (part * G + g) % BS_GROUPS < by_tma;
                    if (lane == 0) mbar_arrive_expect_tx(full, here * 512 * T::CH);
                    __syncwarp();
                }
#pragma unroll
                for (int g = 0; g < G; g++) {
                    const int q = part * G + g;
                    int4 rr = rows[T::BY_LANE ? 0 : g];
                    if (T::BY_LANE)
                        rr = make_int4(__shfl_sync(0xffffffffu, rr.x, g), __shfl_sync(0xffffffffu, rr.y, g), __shfl_sync(0xffffffffu, rr.z, g),
                                       __shfl_sync(0xffffffffu, rr.w, g));
#pragma unroll
                    for (int c = 0; c < T::CH; c++) {
                        if (q % BS_GROUPS < by_tma) {
                            if (lane == 0) tma_gather4(slot(q) + c * T::B_CHUNK_BYTES, &tmap_rows, n + c * 64, rr, full);
                            continue;
                        }
                        const int row_in = lane >> 3, piece = lane & 7;       // four rows x eight 16-byte pieces
                        const int row = row_in == 0 ? rr.x : row_in == 1 ? rr.y : row_in == 2 ? rr.z : rr.w;
                        const int rs = q % BS_GROUPS * 4 + row_in, col = n + c * 64 + piece * 8;
                        const bool ok = col < p.N && row < p.K;               // N % 8 == 0: a piece lies entirely inside or outside
                        cp_async_16_zfill(smem_u32(st) + (uint32_t)(q / BS_GROUPS * T::B_BLOCK_BYTES + c * T::B_CHUNK_BYTES + rs * 128 + ((piece ^ (rs & 7)) << 4)),
                                          ok ? p.B + (size_t)row * p.ldb + col : p.B, ok ? 16u : 0u);
                    }
                }
                cp_async_mbar_arrive_noinc(full);   // arrives once this lane's copies have landed
            }
            ++issued;
        }
        if (gmode == GATHER_CPASYNC) cp_async_wait_all();
        if (lane == 0 && issued > 0) atomicMax(b_fills, first + (issued - 1) * ng + 1);
        __syncwarp();
    } else if (warp == T::A_WARP) {
        // ---------------- A producer ----------------
        if (lane == 0) {
            int it = 0, s = 0;
            uint32_t ph = 1;
            bool alive = true;
            for (int tile = blockIdx.x; alive && tile < p.total_tiles; tile += gridDim.x) {
                int mt, n0_unused, slices_unused;
                locate_tile(tile, &mt, &n0_unused, &slices_unused);
                const uint8_t *src = p.am + (size_t)mt * p.ktiles * AM_BLOCK_BYTES;
                for (int kt = 0; kt < p.ktiles; ++kt, ++it) {
                    if (!wait_quiet(&a_free[s], ph, abort_flag, p.status, DEV_TIMEOUT_PRODUCER)) { alive = false; break; }
                    mbar_arrive_expect_tx(&a_full[s], AM_BLOCK_BYTES);
                    bulk_g2s(a_ring + s * AM_BLOCK_BYTES, src + (size_t)kt * AM_BLOCK_BYTES, AM_BLOCK_BYTES, &a_full[s]);
                    if (++s == SA) { s = 0; ph ^= 1; }
                }
            }
            if (*abort_flag) {
                for (int k = it > SA ? it - SA : 0; k < it; ++k) drain_slot(&a_full[k % SA], (uint32_t)(k / SA) & 1u, p.status);
            }
        }
        __syncwarp();
    } else if (warp == T::MMA_WARP) {
        // ---------------- MMA issuer ----------------
        // One elected lane (not lane 0 of a divergent branch: behind elect.sync the compiler keeps descriptors in uniform
        // registers, otherwise every MMA costs 161 clocks to issue, more than it takes to execute).  The tensor pipe queues
        // about two MMAs, so the wait for a stage sits directly in front of its MMAs, where it hides behind the previous stage's.
        if (elect_one()) {
            const uint32_t idesc_full = make_idesc_f16(TILE_M, BN, true, 0u, true);
            const uint32_t idesc_cut = T::CAN_CUT ? make_idesc_f16(TILE_M, BN / 2, true, 0u, true) : idesc_full;
            // descriptor templates: only the start-address field (low 14 bits, in 16-byte units) varies
            const uint64_t adesc0 = make_smem_desc(smem_u32(a_ring), 16, 1024, 2);
            const uint64_t mdesc0 = make_smem_desc(smem_u32(a_ring) + A_IMG_BYTES, 0, 128, 0);
            const uint64_t bdesc0 = make_smem_desc(smem_u32(b_ring), T::B_CHUNK_BYTES, 1024, 2);
            int sa = 0, sb = 0, set = 0;
            uint32_t pa = 0, pb = 0;
            bool alive = true;
            for (int ti = 0; alive && ti < my_tiles; ++ti) {
                const int aset = T::ACCS == 1 ? 0 : ti & 1;
                const uint32_t acc = tmem_base + (uint32_t)(aset * BN);
                const uint32_t idesc0 = (int)blockIdx.x + ti * (int)gridDim.x >= cut_from ? idesc_cut : idesc_full;
                // the epilogue must have read this accumulator's previous tile
                if (!wait_one(&acc_empty[aset], ((uint32_t)(T::ACCS == 1 ? ti : ti >> 1) & 1u) ^ 1u, abort_flag, p.status, DEV_TIMEOUT_MMA)) break;
                for (int kt = 0; kt < p.ktiles; ++kt) {
                    const uint32_t mcol = tmem_base + (uint32_t)(T::META_COL + set * 4);
                    const uint32_t aoff = (uint32_t)(sa * AM_BLOCK_BYTES) >> 4;
                    if (!wait_one(&a_full[sa], pa, abort_flag, p.status, DEV_TIMEOUT_MMA)) { alive = false; break; }
                    tc_fence_after();
                    // metadata image: 128 rows x 16 bytes, 8-row core matrices stored back to back
                    tc_cp_128x128b(mcol, mdesc0 + aoff);
#pragma unroll
                    for (int kb = 0; kb < STAGES_PER_KT; ++kb) {   // K=32 blocks of the k-tile, one B stage each
                        if (!wait_one(&b_full[sb], pb, abort_flag, p.status, DEV_TIMEOUT_MMA)) { alive = false; break; }
                        if (gmode == GATHER_CPASYNC) fence_proxy_async();  // per-thread copies are read by the tensor core's proxy
                        tc_fence_after();
                        const uint32_t boff = (uint32_t)(sb * T::B_STAGE_BYTES) >> 4;
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
                            // A: K-major, 128-byte swizzle, 8-row groups 1024 B apart; one MMA reads 32 B of each row.
                            // B: N-major, 128-byte swizzle; 8 gathered rows = 1024 B, next 64 columns = one slice further.
                            tc_mma_sp_f16(acc, adesc0 + aoff + (uint32_t)(kb * 32 >> 4), bdesc0 + boff + (uint32_t)(b * T::B_BLOCK_BYTES >> 4),
                                          mcol + (uint32_t)(kb & ~1), idesc0 | (uint32_t)(kb & 1), (kt | kb) != 0 ? 1u : 0u, mk[0], mk[1], mk[2], mk[3]);
                        }
                        tc_commit(&b_free[sb]);
                        if (++sb == SB) { sb = 0; pb ^= 1; }
                    }
                    if (!alive) break;
                    tc_commit(&a_free[sa]);
                    if (kt == p.ktiles - 1) tc_commit(&acc_full[aset]);
                    if (++sa == SA) { sa = 0; pa ^= 1; }
                    set = set + 1 == T::META_SETS ? 0 : set + 1;
                }
            }
        }
        __syncwarp();
    } else if (warp >= T::EPI_WARP0) {
        // ---------------- epilogue ----------------
        constexpr int PART = T::PART;
        const int grp = (warp - T::EPI_WARP0) >> 2;     // one accumulator: drains its half of every tile's columns; two: the tiles ti with ti & 1 == grp
        const int q = warp & 3;                         // tensor-memory lane quadrant this warp may read
        const int arow = mma_row_to_actual(q * 32 + lane);
        const bool leader = ((warp - T::EPI_WARP0) & 3) == 0 && lane == 0;
        uint8_t *stg = out_ring + grp * T::OUT_STAGE_BYTES;
        const uint32_t trow = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(T::ACCS == 1 ? 0 : grp * BN);
        for (int ti = T::ACCS == 1 ? 0 : grp; ti < my_tiles; ti += T::ACCS) {
            const int tile = (int)blockIdx.x + ti * (int)gridDim.x;
            int mt, n0, slices;
            locate_tile(tile, &mt, &n0, &slices);
            const int aset = T::ACCS == 1 ? 0 : grp;
            // with stores through shared memory the four warps of a group leave the loop together (they meet at named barriers below)
            const bool got = wait_warp(&acc_full[aset], (uint32_t)(T::ACCS == 1 ? ti : ti >> 1) & 1u, abort_flag, p.status, DEV_TIMEOUT_EPILOGUE);
            if (p.tma_out ? !named_barrier_and(1 + grp, 128, got) : !got) break;
            tc_fence_after();
            auto release = [&] {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[aset]);
            };
            // This group's columns.  With one accumulator the MMAs of the next tile wait until the last column has been read, but the loads
            // go on: the rings hold what arrives in that time, and the MMAs are more than twice as fast as the loads.
            const int mine = T::DRAIN / T::CH * slices, first = T::ACCS == 1 ? grp * mine : 0;
            const uint32_t tacc = trow + (uint32_t)first;
            n0 += first;
            if (!p.tma_out) {
                if (mine == T::DRAIN) {
                    if (p.layout == 0) store_tile<T::DRAIN, false>(TileStoreMN(tacc, q, (int64_t)mt * TILE_M, n0, p), release);
                    else store_tile<T::DRAIN, false>(TileStoreNM(tacc, q, (int64_t)mt * TILE_M, n0, p), release);
                } else if (T::CAN_CUT) {   // half a tile
                    if (p.layout == 0) store_tile<64, false>(TileStoreMN(tacc, q, (int64_t)mt * TILE_M, n0, p), release);
                    else store_tile<64, false>(TileStoreNM(tacc, q, (int64_t)mt * TILE_M, n0, p), release);
                }
                continue;
            }
            // [N,M] (+ bias) to several destinations (peers' buffers), or on request: parts of PART rows (n) x 128 columns (m) go
            // through shared memory and leave with one TMA store per destination, 256 contiguous bytes a row
            const int64_t row = (int64_t)mt * TILE_M + arow;
            const bool has_bias = p.bias != nullptr;
            const __half bias = (has_bias && row < p.M) ? p.bias[row] : __ushort_as_half((unsigned short)0);
#pragma unroll 1
            for (int part = 0; part < mine / PART; part += 2) {
                // two parts are read at a time, so that the MMAs of the next tile wait for the stores of all but the last two (two destinations, 3456 x 1072,
                // 128:2:16, N = 2224 16.9 -> 15.9 us, 5248 x 5280, 128:2:32, N = 8016 92.1 -> 88.9)
                __half2 held[2][PART / 2];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    uint32_t v[PART / 8][8];
#pragma unroll
                    for (int i = 0; i < PART / 8; i++) tc_ld_32x32b_x8(tacc + (uint32_t)((part + h) * PART + 8 * i), v[i]);
                    tc_wait_ld();
#pragma unroll
                    for (int c = 0; c < PART; c += 2) held[h][c / 2] = __floats2half2_rn(__uint_as_float(v[c / 8][c % 8]), __uint_as_float(v[c / 8][c % 8 + 1]));
                }
                if (part == mine / PART - 2) release();
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    if (leader) bulk_wait_group_read0();   // the previous store has finished reading the staging buffer
                    named_barrier_sync(1 + grp, 128);
                    __half *col = reinterpret_cast<__half *>(stg) + arow;
#pragma unroll
                    for (int c = 0; c < PART; c += 2) {
                        __half2 x = held[h][c / 2];
                        if (has_bias) x = __hadd2(x, __half2half2(bias));
                        col[c * TILE_M] = __low2half(x);
                        col[(c + 1) * TILE_M] = __high2half(x);
                    }
                    fence_proxy_async();
                    named_barrier_sync(1 + grp, 128);
                    const int nbase = n0 + (part + h) * PART;
                    if (leader && nbase < p.N) {
                        tma_store_2d(&tmap_out, stg, mt * TILE_M, nbase);
                        for (int d = 1; d < p.n_out; d++) tma_store_2d(&more_out.m[d - 1], stg, mt * TILE_M, nbase);
                        bulk_commit_group();
                    }
                }
            }
        }
        if (leader) bulk_wait_group_read0();  // the stores have read shared memory (their global writes complete with the grid)
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 0 && *abort_flag) drain_ring(b_full, SB, *b_fills, p.status);
    if (warp == T::MMA_WARP) {
        tc_fence_after();
        tmem_dealloc(tmem_base, T::TMEM_COLS);
    }
}

template <int BN, int NB>
cudaError_t set_attr()
{
    return cudaFuncSetAttribute(spmm_kernel<BN, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, Traits<BN, NB>::SMEM_BYTES);
}

template <int BN, int NB>
cudaError_t launch_one(const SpmmConfig &cfg, const CUtensorMap &tmap_rows, const CUtensorMap &tmap_tile, const CUtensorMap &tmap_out,
                       const OutMaps &more_out, const SpmmParams &p, cudaStream_t stream)
{
    using T = Traits<BN, NB>;
    cudaLaunchConfig_t lc = {};
    cudaLaunchAttribute attr = early_launch();
    lc.gridDim = dim3((unsigned)cfg.grid, 1, 1);
    lc.blockDim = dim3(T::NUM_THREADS, 1, 1);
    lc.dynamicSmemBytes = T::SMEM_BYTES;
    lc.stream = stream;
    lc.attrs = &attr;
    lc.numAttrs = 1;
    return cudaLaunchKernelEx(&lc, spmm_kernel<BN, NB>, tmap_rows, tmap_tile, tmap_out, more_out, p, cfg.cut_from);
}

int g_num_sms = 0;

}  // namespace

// A last wave that fills at most half of the SMs has its tiles cut in two (V = 128 and 64, gather4 only: the ablations load whole stages).  Half a
// tile takes 0.65 of the time of a whole one, bound by the latency of its half-filled stages; quarters take as long as halves.  [K,N] to
// [M,N], us, many calls (after a pause), whole and cut:  12288 x 12288, V = 128, m = 16, N = 2048 (28 tiles beyond five waves) 131.7 (121.1), 129.3 (116.7);
// 4096 x 12288, m = 8, N = 4096 (68 beyond three) 165.9 (152.8), 160.5 (144.1);  12288 x 12288, V = 64, m = 32, N = 2048 (56 beyond ten) 114.6
// (110.9), 113.0 (108.7).  More than half (124 beyond 13 waves, 4096 x 4096, m = 8, N = 16384), which makes two waves of halves: 217.0, 221.2.
//
// The estimate, in us: start-up and last epilogue, then per wave a k-tile's time (0.76 us: 1340 clocks at the 1760 MHz of a call among many) and what a tile
// change costs.  Calls among many take 0.93 to 1.16 of it (ten sizes from 62 us to 14 ms, V = 128, 64 and 32; after a pause less, at the full clock).  With
// boxes of rows instead of gathers (m = 4) a line of its own for each V, fitted to 168 sizes of 512 to 12288 rows and k and 256 to 16384 columns: between this
// kernel and the one for few tiles the faster one is taken but for 1.08 of its time at most beyond 12 us.  (With the cost of gathers up to 1.72: 4096 x 4096,
// 128:2:4, N = 16384 took 565 us in the other kernel and takes 333 in this one.)
//
// Tile configurations: V=128 -> one block per tile, BN 256; V=64 -> two blocks, BN 128; V=32 -> four blocks, BN 64 (NB * BN = 256:
// every B stage is 16 KiB).
float spmm_select_config(int V, int N, int M, int ktiles, int max_ctas, int gather_mode, SpmmConfig *cfg)
{
    const int mtiles = (M + TILE_M - 1) / TILE_M;
    cfg->stages = GATHER_PRODUCER_WARPS;
    cfg->threads = Traits<256, 1>::NUM_THREADS;
    cfg->part = Traits<256, 1>::PART;
    if (V == 128) {
        cfg->bn = 256; cfg->nb = 1; cfg->smem_bytes = Traits<256, 1>::SMEM_BYTES;
    } else if (V == 64) {
        cfg->bn = 128; cfg->nb = 2; cfg->smem_bytes = Traits<128, 2>::SMEM_BYTES;
    } else if (V == 32) {
        cfg->bn = 64; cfg->nb = 4; cfg->smem_bytes = Traits<64, 4>::SMEM_BYTES;
    } else {
        return -1.0f;
    }
    const long long tiles = (long long)mtiles * ((N + cfg->bn - 1) / cfg->bn);
    int sms = g_num_sms > 0 ? g_num_sms : 148;
    if (max_ctas > 0 && max_ctas < sms) sms = max_ctas;  // the caller keeps some SMs free (e.g. for a collective that runs beside the product)
    const long long waves = tiles / sms;
    const int rest = (int)(tiles - waves * sms);
    const bool cut = gather_mode == GATHER_TMA4 && cfg->bn > 64 && rest > 0 && 2 * rest <= sms;
    cfg->tiles = (int)tiles + (cut ? rest : 0);
    cfg->cut_from = cut ? (int)(waves * sms) : cfg->tiles;
    cfg->grid = cfg->tiles < sms ? cfg->tiles : sms;
    if (gather_mode == GATHER_CONTIG) {
        static const float kt_us[3] = {0.58f, 0.645f, 0.76f}, tile_us[3] = {1.9f, 0.8f, 0.3f};   // 1, 2 and 4 vector blocks
        const int i = V == 128 ? 0 : V == 64 ? 1 : 2;
        return 4.6f + (float)(waves + (rest != 0)) * (ktiles * kt_us[i] + tile_us[i]);
    }
    return 5.5f + ((float)waves + (rest == 0 ? 0.0f : cut ? 0.65f : 1.0f)) * (V == 128 ? ktiles * 0.76f + 1.7f : ktiles * 0.68f + 1.35f);
}

cudaError_t spmm_init_kernels()
{
    cudaError_t e;
    if ((e = set_attr<256, 1>()) != cudaSuccess) return e;
    if ((e = set_attr<128, 2>()) != cudaSuccess) return e;
    if ((e = set_attr<64, 4>()) != cudaSuccess) return e;
    int dev = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    return cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
}

cudaError_t launch_spmm(const SpmmConfig &cfg, const CUtensorMap &tmap_rows, const CUtensorMap &tmap_tile, const CUtensorMap &tmap_out,
                        const OutMaps &more_out, const SpmmParams &p, cudaStream_t stream)
{
    if (cfg.nb == 1) return launch_one<256, 1>(cfg, tmap_rows, tmap_tile, tmap_out, more_out, p, stream);
    if (cfg.nb == 2) return launch_one<128, 2>(cfg, tmap_rows, tmap_tile, tmap_out, more_out, p, stream);
    if (cfg.nb == 4) return launch_one<64, 4>(cfg, tmap_rows, tmap_tile, tmap_out, more_out, p, stream);
    return cudaErrorInvalidValue;
}

}  // namespace vnm
