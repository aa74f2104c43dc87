// twm_dense_experts_tc.cuh — the grouped product of many rows an expert on pairs of SMs: C[row][N] = A[row][K] . W[expert of the row][N][K]^T.
//
// The pair of CTAs and its stages are those of twm_dense_tc2.cuh with the operands' parts changed: 256 WEIGHT rows are the MMA's rows, and
// up to 256 of an expert's activation rows its columns.  An expert's weight rows fill whole tiles; its activation rows, of any number, are
// spread evenly over the fewest tiles and rounded up to 32, so little is multiplied for rows that are not there (128 x 256 tiles with
// activations as rows round up to 128: an eighth more at 512 rows an expert, and the pair's 256 rows a quarter).  Below 128 rows an expert
// bound by reading the weights.  64 experts of 2048 x 1024, 512 rows each on average: 147.8 us on one SM's tiles, 120.9 to 129.9 this way, 0.64 to
// 0.69 of the GEMM rate: the tensor pipe is busy 67 % of the time (72 % of the time that an SM has a tile) and DRAM 47 % (every operand is read
// once), so neither is what bounds it yet.  A prompt of 4096 tokens on 16 layers of them: 11.57 -> 11.03 ms.
//
// Read-back: thread = output column (its TMEM lane), 16 activation rows at a time; neighbouring threads exchange halves, so that a warp
// stores 64 contiguous bytes of two rows.
#pragma once

#include "twm_dense_tc2.cuh"

namespace twm {
namespace dense {

constexpr int EX_TOKENS = 256, EX_STEP = 32;                 // activation rows a tile: at most, and in multiples of

template <int EPI>
__global__ void __launch_bounds__(TC_THREADS, 1)
gemm_experts_kernel(const __grid_constant__ TcArgs g)
{
    using C = Tc2Cfg<EX_TOKENS>;
    constexpr int STAGES = C::STAGES;
    extern __shared__ uint8_t tc_smem_raw[];
    uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t full[STAGES], empty[STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_s;
    __shared__ int abort_s;
    __shared__ int pre[MOE_MAX_EXPERTS + 1];                 // the tiles ahead of each expert's
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
    if (warp == 0) {
        pdl_wait_prior_grids();
        warp_prefix([&](int e) { return (g.offsets[e + 1] - g.offsets[e] + EX_TOKENS - 1) / EX_TOKENS * g.n_tiles; }, g.experts, pre, lane);
    }
    __syncthreads();
    cluster_sync_all();                                      // the other CTA's barriers are ready as well
    tc::tc_fence_after();
    pdl_launch_dependents();
    const uint32_t tmem = tmem_s;
    const int tiles = pre[g.experts];
    // tile t: its first activation row, how many the MMA takes and how many there are, its first output column and weight row
    struct Tile { int row, take, rows, n, w; };
    auto tile_at = [&](int t) {
        Tile x;
        const int e = prefix_find(pre, g.experts, t), mt = (pre[e + 1] - pre[e]) / g.n_tiles, i = t - pre[e];
        const int first = g.offsets[e], count = g.offsets[e + 1] - first, nt = i / mt;
        x.take = ((count + mt - 1) / mt + EX_STEP - 1) / EX_STEP * EX_STEP;
        x.row = first + (i - nt * mt) * x.take;
        x.rows = min(x.take, first + count - x.row);
        x.n = nt * 2 * TC_BM;
        x.w = e * g.N + x.n;
        return x;
    };

    if (warp == TC_WARP_TMA) {
        if (elect_one()) {
            pdl_wait_prior_grids();
            int it = 0;
            bool ok = true;
            for (int t = pair; t < tiles && ok; t += pairs) {
                const Tile x = tile_at(t);
                for (int kk = 0; kk < k_steps; ++kk, ++it) {
                    const int slot = it % STAGES;
                    if (it >= STAGES && !mbar_wait_bounded(&empty[slot], ((it / STAGES) - 1) & 1, abort_flag)) { ok = false; break; }
                    // the leader announces both CTAs' bytes on its barrier.  Boxes are whole: rows past the tile's enter nothing that is stored
                    if (rank == 0) mbar_arrive_expect_tx(&full[slot], 2u * C::STAGE_BYTES);
                    const uint32_t bar = mapa_shared(smem_u32(&full[slot]), 0);
                    uint8_t* dst = ring + (size_t)slot * C::STAGE_BYTES;
                    tma_load_2d_pair(dst, &g.w_map, kk * TC_BK, x.w + rank * TC_BM, bar);
                    tma_load_2d_pair(dst + TC_A_BYTES, &g.a_map, kk * TC_BK, x.row + rank * (x.take / 2), bar);
                }
            }
        }
        __syncwarp();
    } else if (warp == TC_WARP_MMA) {
        if (rank == 0 && elect_one()) {
            int it = 0, nt = 0;
            bool ok = true;
            for (int t = pair; t < tiles && ok; t += pairs, ++nt) {
                const Tile x = tile_at(t);
                // D f32, A and B bf16, both K-major, 256 x take over the pair
                const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(x.take >> 3) << 17) | ((uint32_t)(2 * TC_BM >> 4) << 24);
                const int acc = nt & 1;
                if (nt >= 2 && !mbar_wait_bounded(&acc_empty[acc], ((nt >> 1) - 1) & 1, abort_flag)) { ok = false; break; }
                tc::tc_fence_after();
                for (int kk = 0; kk < k_steps; ++kk, ++it) {
                    const int slot = it % STAGES;
                    if (!mbar_wait_bounded(&full[slot], (it / STAGES) & 1, abort_flag)) { ok = false; break; }
                    tc::tc_fence_after();
                    const uint32_t base = smem_u32(ring + (size_t)slot * C::STAGE_BYTES);
                    uint64_t wd = sw128_desc(base), ad = sw128_desc(base + TC_A_BYTES);
#pragma unroll
                    for (int h = 0; h < TC_BK / 16; ++h) {
                        mma_pair(tmem + acc * 256, wd, ad, idesc, (kk == 0 && h == 0) ? 0u : 1u);
                        wd += 2;
                        ad += 2;
                    }
                    commit_pair(&empty[slot]);
                }
                if (ok) commit_pair(&acc_full[acc]);
            }
        }
        __syncwarp();
    } else {
        const bool pairwise = EPI != TWM_EPI_STORE_F32 && ((g.ldc | g.N) & 1) == 0 && (reinterpret_cast<uintptr_t>(g.c) & 3) == 0;
        int nt = 0;
        for (int t = pair; t < tiles; t += pairs, ++nt) {
            const Tile x = tile_at(t);
            const int acc = nt & 1;
            if (!tc::wait_uniform(&acc_full[acc], (nt >> 1) & 1, abort_flag)) break;
            tc::tc_fence_after();
            const int n = x.n + rank * TC_BM + warp * 32 + lane;
            const uint32_t at = tmem + ((uint32_t)(warp * 32) << 16) + acc * 256;
#pragma unroll 1
            for (int c0 = 0; c0 < x.rows; c0 += 16) {
                uint32_t d[16];
                float v[16];
                tc::tmem_ld<16>(at + c0, d);
                tc::tmem_wait_ld();
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = epilogue_value<EPI>(__uint_as_float(d[j]));
                if (EPI == TWM_EPI_STORE_F32) {
                    float* to = reinterpret_cast<float*>(g.c) + (size_t)(x.row + c0) * g.ldc + n;
#pragma unroll
                    for (int j = 0; j < 16; ++j) if (n < g.N && c0 + j < x.rows) to[(size_t)j * g.ldc] = v[j];
                } else if (pairwise) {
                    // even threads keep row j of two columns, odd ones row j + 1
                    bf16* to = reinterpret_cast<bf16*>(g.c) + (size_t)(x.row + c0 + (lane & 1)) * g.ldc + (n & ~1);
#pragma unroll
                    for (int j = 0; j < 16; j += 2) {
                        const float other = __shfl_xor_sync(0xffffffffu, lane & 1 ? v[j] : v[j + 1], 1);
                        const __nv_bfloat162 two = lane & 1 ? __floats2bfloat162_rn(other, v[j + 1]) : __floats2bfloat162_rn(v[j], other);
                        if (n < g.N && c0 + j + (lane & 1) < x.rows) *reinterpret_cast<__nv_bfloat162*>(to + (size_t)j * g.ldc) = two;
                    }
                } else {
                    bf16* to = reinterpret_cast<bf16*>(g.c) + (size_t)(x.row + c0) * g.ldc + n;
#pragma unroll
                    for (int j = 0; j < 16; ++j) if (n < g.N && c0 + j < x.rows) to[(size_t)j * g.ldc] = __float2bfloat16_rn(v[j]);
                }
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
