// twm_dense_tc2.cuh — the product of twm_dense_tc.cuh with two SMs on one tile, for many rows.
//
// One SM's 128 x 256 tile is bound by its shared memory: 48 KB come in and go out again per 512 clocks of
// MMA.  Here a pair of CTAs (one cluster) computes 256 x 256: each loads its own 128 activation rows and
// HALF of the weight rows (256 columns: 32 KB a stage, six stages; 224 and 192: 30 and 28 KB, seven), the tensor cores of the pair share the halves
// (tcgen05.mma.cta_group::2, M = 256), and each CTA ends up with its 128 rows of the result in its own
// tensor memory.  The leader's MMA thread issues for both; both CTAs' loads count on the leader's barriers;
// a commit tells both when a stage is free and when an accumulator is complete.  A gated product takes
// its gate rows through the leader and its up rows through the other CTA.  No load is multicast.
//
// BN: 256 columns a tile, or 224 or 192 where those fill the last wave of the pairs better (tc_tile_choice): 3584 columns of 2048 rows
// are 112 tiles of 256 x 256, two waves of 74 pairs, and 128 of 256 x 224, two waves of shorter ones.
#pragma once

#include "twm_dense_tc.cuh"

namespace twm {
namespace dense {

template <int BN>
struct Tc2Cfg {
    static constexpr int STAGE_BYTES = TC_A_BYTES + BN / 2 * TC_BK * 2;              // per CTA: 128 activation rows, half the weight rows
    static constexpr int STAGES = BN == 256 ? 6 : 7;
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024;
    static constexpr uint32_t TMEM_COLS = 512;                                      // two accumulators, 256 columns apart
};

__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* map, int x, int y, uint32_t cluster_bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(cluster_bar)
        : "memory");
}
__device__ __forceinline__ void mma_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// arrives on the barrier at this offset in both CTAs of the pair once the MMAs issued so far are complete
__device__ __forceinline__ void commit_pair(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}

template <int BN, int EPI>
__global__ void __launch_bounds__(TC_THREADS, 1)
gemm_tc2_kernel(const __grid_constant__ TcArgs g)
{
    constexpr bool GATED = EPI == TWM_EPI_GELU_GLU;
    constexpr int OUT = GATED ? BN / 2 : BN;                 // output columns per tile
    using C = Tc2Cfg<BN>;
    constexpr int STAGES = C::STAGES;
    extern __shared__ uint8_t tc_smem_raw[];
    uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t full[STAGES], empty[STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_s;
    __shared__ int abort_s;
    volatile int* abort_flag = &abort_s;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = (int)cluster_ctarank();                 // 0 = leader
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int k_steps = (g.K + TC_BK - 1) / TC_BK;

    if (tid == 0) {
        prefetch_map(&g.a_map);
        prefetch_map(&g.w_map);
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 8); }
        abort_s = 0;
        mbar_fence_init();
    }
    if (warp == TC_WARP_MMA) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_s)), "r"(C::TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        tc::tc_fence_before();
    }
    __syncthreads();
    cluster_sync_all();                                      // the other CTA's barriers are ready as well
    tc::tc_fence_after();
    pdl_launch_dependents();
    const uint32_t tmem = tmem_s;
    const int tiles = g.m_tiles * g.n_tiles;
    // tile t: the first row of this CTA's half, and its column tile
    struct Tile { int row, n; };
    auto tile_at = [&](int t) {
        Tile x;
        int m;
        tc_tile(t, g.m_tiles, g.n_tiles, m, x.n);
        x.row = m * 2 * TC_BM + rank * TC_BM;
        return x;
    };

    if (warp == TC_WARP_TMA) {
        if (elect_one()) {
            // the leader announces both CTAs' bytes on its barrier; a load of the other CTA that is faster only runs the count ahead
            auto load_w = [&](int slot, const Tile& x, int kk) {
                if (rank == 0) mbar_arrive_expect_tx(&full[slot], 2u * C::STAGE_BYTES);
                const int row = GATED ? (rank == 0 ? x.n * OUT : g.N + x.n * OUT) : x.n * OUT + rank * (BN / 2);
                tma_load_2d_pair(ring + (size_t)slot * C::STAGE_BYTES + TC_A_BYTES, &g.w_map, kk * TC_BK, row, mapa_shared(smem_u32(&full[slot]), 0));
            };
            auto load_a = [&](int slot, const Tile& x, int kk) {
                tma_load_2d_pair(ring + (size_t)slot * C::STAGE_BYTES, &g.a_map, kk * TC_BK, x.row, mapa_shared(smem_u32(&full[slot]), 0));
            };
            int it = 0;
            bool ok = true;
            const int early = min(STAGES, k_steps);
            const Tile first = tile_at(pair);                // the host launches no more pairs than tiles
            for (int kk = 0; kk < early; ++kk) load_w(kk, first, kk);
            pdl_wait_prior_grids();
            for (int kk = 0; kk < early; ++kk) load_a(kk, first, kk);
            for (int t = pair; t < tiles && ok; t += pairs) {
                const Tile x = tile_at(t);
                for (int kk = 0; kk < k_steps; ++kk, ++it) {
                    if (it < early) continue;
                    const int slot = it % STAGES;
                    if (it >= STAGES && !mbar_wait_bounded(&empty[slot], ((it / STAGES) - 1) & 1, abort_flag)) { ok = false; break; }
                    load_w(slot, x, kk);
                    load_a(slot, x, kk);
                }
            }
        }
        __syncwarp();
    } else if (warp == TC_WARP_MMA) {
        if (rank == 0 && elect_one()) {
            // D f32, A and B bf16, both K-major, 256 x BN over the pair
            constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(2 * TC_BM >> 4) << 24);
            int it = 0, nt = 0;
            bool ok = true;
            for (int t = pair; t < tiles && ok; t += pairs, ++nt) {
                const int acc = nt & 1;
                if (nt >= 2 && !mbar_wait_bounded(&acc_empty[acc], ((nt >> 1) - 1) & 1, abort_flag)) { ok = false; break; }
                tc::tc_fence_after();
                for (int kk = 0; kk < k_steps; ++kk, ++it) {
                    const int slot = it % STAGES;
                    if (!mbar_wait_bounded(&full[slot], (it / STAGES) & 1, abort_flag)) { ok = false; break; }
                    tc::tc_fence_after();
                    const uint32_t base = smem_u32(ring + (size_t)slot * C::STAGE_BYTES);
                    uint64_t ad = sw128_desc(base), bd = sw128_desc(base + TC_A_BYTES);
#pragma unroll
                    for (int h = 0; h < TC_BK / 16; ++h) {
                        mma_pair(tmem + acc * 256, ad, bd, idesc, (kk == 0 && h == 0) ? 0u : 1u);
                        ad += 2;
                        bd += 2;
                    }
                    commit_pair(&empty[slot]);
                }
                if (ok) commit_pair(&acc_full[acc]);
            }
        }
        __syncwarp();
    } else {
        // read-back: thread = row (its TMEM lane) of this CTA's half, 16 columns at a time
        int nt = 0;
        for (int t = pair; t < tiles; t += pairs, ++nt) {
            const Tile x = tile_at(t);
            const int acc = nt & 1;
            if (!tc::wait_uniform(&acc_full[acc], (nt >> 1) & 1, abort_flag)) break;
            tc::tc_fence_after();
            const int row = x.row + warp * 32 + lane;
            const size_t row_off = (size_t)row * g.ldc;
            const uint32_t at = tmem + ((uint32_t)(warp * 32) << 16) + acc * 256;
#pragma unroll 1
            for (int c0 = 0; c0 < OUT; c0 += 16) {
                uint32_t d[16];
                float v[16];
                tc::tmem_ld<16>(at + c0, d);
                if (GATED) {
                    uint32_t u[16];
                    tc::tmem_ld<16>(at + OUT + c0, u);
                    tc::tmem_wait_ld();
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = gelu_tanh(__uint_as_float(d[j])) * __uint_as_float(u[j]);
                } else {
                    tc::tmem_wait_ld();
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(d[j]);
                }
                if (row < g.M && x.n * OUT + c0 < g.N) tc_store16<EPI>(g.c, row_off, x.n * OUT + c0, g.N, v);
            }
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(&acc_empty[acc]), 0));
        }
    }
    tc::tc_fence_before();
    __syncthreads();
    cluster_sync_all();                                      // nobody leaves while the pair's MMAs or arrivals may touch its memory
    if (warp == TC_WARP_MMA) {
        tc::tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::TMEM_COLS) : "memory");
    }
}

}  // namespace dense
}  // namespace twm
