// twm_dense_tcs.cuh — C[M][N] = A[M][K] . W[N][K]^T in bfloat16 on the tensor cores, for products of few tiles: one CTA a tile, or a
// cluster of up to eight CTAs that share K.
//
// Bound by reading W; before that by what one SM can take in (64 bytes a clock, activations included) where fewer tiles than SMs
// leave the machine idle: the down product of a 2048-wide layer has 32 tiles of 64 columns.  The rows are spread evenly over the
// row tiles (333 rows: three tiles of 112), and a stage holds no more of them: fewer bytes a stage, more stages.  Each CTA
// of a cluster accumulates its share of K in TMEM and leaves the sums in its shared memory, where the stages were; each adds up its
// share of the rows over the cluster in rank order: the same result every time, no workspace.
//
// A chain of calls in a graph, weights cold, against twm_dense_tc.cuh: 2048 x 8192, 100 rows: 27.2 -> 12.1 us (K over four), 333 rows:
// 27.6 -> 19.7; 3584 x 18944, 100 rows: 58.6 -> 29.1 us (4.7 TB/s); 2048 x 2048, 100 rows: 10.2 -> 8.0; 5120 x 2048, 2 rows: 15.0 -> 8.7;
// a router's 64 x 2048, 4096 rows: 9.6 -> 7.2, and its error against 64 bits 2.1e-6 -> 4.7e-7 of the results: the tensor core cuts
// when it adds, and a share of K is a shorter sum.  Tiles of 256 columns
// gained only at 333 rows x 3584 x 18944 (51 instead of 62 us) and lost elsewhere, half the stages with two CTAs to an SM
// lost wherever one CTA an SM is enough.
#pragma once

#include "twm_dense_tc.cuh"

namespace twm {
namespace dense {

constexpr int TS_MAX_SPLITS = 8, TS_MAX_STAGES = 8;

struct TcsArgs {
    void* c;
    int ldc, M, N, K;               // gated: N output columns, 2 N weight rows
    int m_tiles, bm;                // rows a tile, a multiple of 8 up to 128: the rows spread evenly over the tiles
    int splits, stages;
    alignas(64) CUtensorMap a_map;  // bf16 [M][K], box 64 x bm
    alignas(64) CUtensorMap w_map;  // bf16 [rows][K], box 64 x BN (gated: 64 x BN/2)
};

template <int BN>
__host__ __device__ constexpr int ts_stage_bytes(int bm) { return (bm + BN) * TC_BK * 2; }
template <int BN>
__host__ __device__ constexpr int ts_sum_bytes() { return TC_BM * (BN + 4) * 4; }
// the stages, what the last stage's MMA reads past its rows, and where the sums of the cluster come together
template <int BN>
size_t ts_smem_bytes(int bm, int stages, int splits)
{
    const int ring = stages * ts_stage_bytes<BN>(bm) + (TC_BM - bm) * TC_BK * 2;
    return 1024 + (splits > 1 ? std::max(ring, ts_sum_bytes<BN>()) : ring);
}

template <int EPI>
__device__ __forceinline__ void tc_store4(void* c, size_t row_off, int n, int N, const float (&v)[4]) {
    if (EPI == TWM_EPI_STORE_F32) {
        float* p = reinterpret_cast<float*>(c) + row_off + n;
        if (n + 4 <= N && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
            *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) if (n + j < N) p[j] = v[j];
        }
    } else {
        bf16* p = reinterpret_cast<bf16*>(c) + row_off + n;
        if (n + 4 <= N && (reinterpret_cast<uintptr_t>(p) & 7) == 0) {
            const __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
            *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) if (n + j < N) p[j] = __float2bfloat16_rn(v[j]);
        }
    }
}

template <int BN, int EPI>
__global__ void __launch_bounds__(TC_THREADS, 2)
gemm_tcs_kernel(const __grid_constant__ TcsArgs g)
{
    constexpr bool GATED = EPI == TWM_EPI_GELU_GLU;
    constexpr int OUT = GATED ? BN / 2 : BN, B_BYTES = BN * TC_BK * 2, LD = BN + 4;
    extern __shared__ uint8_t ts_smem_raw[];
    uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(ts_smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t full[TS_MAX_STAGES], empty[TS_MAX_STAGES], acc_full;
    __shared__ uint32_t tmem_s;
    __shared__ int abort_s;
    volatile int* abort_flag = &abort_s;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = blockIdx.x % g.splits, tile = blockIdx.x / g.splits;
    const int row0 = tile % g.m_tiles * g.bm, n0 = tile / g.m_tiles * OUT, rows = min(g.bm, g.M - row0);
    const int k_tiles = (g.K + TC_BK - 1) / TC_BK;
    const int k_first = (int)((long)rank * k_tiles / g.splits), steps = (int)((long)(rank + 1) * k_tiles / g.splits) - k_first;
    const uint32_t stage_bytes = ts_stage_bytes<BN>(g.bm);

    if (tid == 0) {
        prefetch_map(&g.a_map);
        prefetch_map(&g.w_map);
        for (int s = 0; s < g.stages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(&acc_full, 1);
        abort_s = 0;
        mbar_fence_init();
    }
    if (warp == TC_WARP_MMA) {
        tc::tmem_alloc(&tmem_s, BN);
        tc::tc_fence_before();
    }
    __syncthreads();
    tc::tc_fence_after();
    pdl_launch_dependents();
    if (g.splits > 1) cluster_started();
    const uint32_t tmem = tmem_s;
    bool complete = true;                                           // readers: the sums are

    if (warp == TC_WARP_TMA) {
        if (elect_one()) {
            auto load_w = [&](int slot, int kk) {
                uint8_t* dst = ring + slot * stage_bytes;
                mbar_arrive_expect_tx(&full[slot], stage_bytes);
                tma_load_2d(dst, &g.w_map, (k_first + kk) * TC_BK, n0, &full[slot]);
                if (GATED) tma_load_2d(dst + B_BYTES / 2, &g.w_map, (k_first + kk) * TC_BK, g.N + n0, &full[slot]);
            };
            auto load_a = [&](int slot, int kk) { tma_load_2d(ring + slot * stage_bytes + B_BYTES, &g.a_map, (k_first + kk) * TC_BK, row0, &full[slot]); };
            // the first stages: weights before the wait for the preceding kernel, activations after it
            const int early = min(g.stages, steps);
            for (int kk = 0; kk < early; ++kk) load_w(kk, kk);
            pdl_wait_prior_grids();
            for (int kk = 0; kk < early; ++kk) load_a(kk, kk);
            int slot = 0;
            uint32_t phase = 0;
            for (int kk = early; kk < steps; ++kk) {
                if (!mbar_wait_bounded(&empty[slot], phase, abort_flag)) break;
                load_w(slot, kk);
                load_a(slot, kk);
                if (++slot == g.stages) { slot = 0; phase ^= 1; }
            }
        }
        __syncwarp();
    } else if (warp == TC_WARP_MMA) {
        if (elect_one()) {
            // D f32, A and B bf16, both K-major; rows past bm are the next operand's bytes, in rows of D that nobody reads
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(TC_BM >> 4) << 24);
            int slot = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int kk = 0; kk < steps; ++kk) {
                if (!mbar_wait_bounded(&full[slot], phase, abort_flag)) { ok = false; break; }
                tc::tc_fence_after();
                const uint32_t base = smem_u32(ring + slot * stage_bytes);
                uint64_t ad = sw128_desc(base + B_BYTES), bd = sw128_desc(base);
#pragma unroll
                for (int h = 0; h < TC_BK / 16; ++h) {
                    tcw::mma_ss(tmem, ad, bd, idesc, (kk == 0 && h == 0) ? 0u : 1u);
                    ad += 2;
                    bd += 2;
                }
                tc::tc_commit(&empty[slot]);
                if (++slot == g.stages) { slot = 0; phase ^= 1; }
            }
            if (ok) tc::tc_commit(&acc_full);
        }
        __syncwarp();
    } else {
        complete = tc::wait_uniform(&acc_full, 0, abort_flag);
        tc::tc_fence_after();
    }

    // read-back: thread = row (its TMEM lane), 16 columns at a time
    const uint32_t at = tmem + ((uint32_t)(warp * 32) << 16);
    const bool reader = warp < 4 && warp * 32 < rows;
    if (g.splits == 1) {
        if (reader && complete) {
            const int r = warp * 32 + lane;
            const size_t row_off = (size_t)(row0 + r) * g.ldc;
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
                if (r < rows && n0 + c0 < g.N) tc_store16<EPI>(g.c, row_off, n0 + c0, g.N, v);
            }
        }
    } else {
        // this CTA's MMAs have run: its sums go where its stages were, and each CTA adds up its share of the rows in rank order
        const int own = (rows + g.splits - 1) / g.splits;
        float* sums = reinterpret_cast<float*>(ring);               // [row][LD]
        if (reader) {
            float* to = sums + (warp * 32 + lane) * LD;
#pragma unroll 1
            for (int c0 = 0; c0 < BN; c0 += 16) {
                uint32_t d[16];
                tc::tmem_ld<16>(at + c0, d);
                tc::tmem_wait_ld();
#pragma unroll
                for (int j = 0; j < 16; j += 4)
                    *reinterpret_cast<float4*>(to + c0 + j) = make_float4(__uint_as_float(d[j]), __uint_as_float(d[j + 1]), __uint_as_float(d[j + 2]), __uint_as_float(d[j + 3]));
            }
        }
        const bool all_ok = cluster_meet(abort_flag);
        for (int i = tid; i < own * (OUT / 4) && all_ok; i += TC_THREADS) {
            const int r = i / (OUT / 4), col = (i - r * (OUT / 4)) * 4, m = rank * own + r;
            if (m >= rows || n0 + col >= g.N) continue;
            const float4 x = cluster_sum4(sums + m * LD + col, g.splits);
            float v[4] = {x.x, x.y, x.z, x.w}, u[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            if (GATED) {
                const float4 z = cluster_sum4(sums + m * LD + OUT + col, g.splits);
                u[0] = z.x; u[1] = z.y; u[2] = z.z; u[3] = z.w;
            }
            if (GATED) {
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] = gelu_tanh(v[j]) * u[j];
            }
            tc_store4<EPI>(g.c, (size_t)(row0 + m) * g.ldc, n0 + col, g.N, v);
        }
        cluster_sync_all();                                         // nobody leaves while its sums may still be read
    }
    tc::tc_fence_before();
    __syncthreads();
    if (warp == TC_WARP_MMA) {
        tc::tc_fence_after();
        tc::tmem_dealloc(tmem, BN);
    }
}

}  // namespace dense
}  // namespace twm
