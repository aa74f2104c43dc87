// twm_dense_f32.cuh — C[M][N] = A[M][K] . W[N][K]^T of the 32-bit models for up to eight rows, in FP32 FMAs.
//
// Bound by reading W.  Tile 8 rows x 128 weight rows, 32 K a stage, three stages of 16-byte asynchronous copies, two CTAs to an SM.
// A thread has one row x 4 weight rows' sums, each as a PAIR over even and odd K
// (fma.rn.f32x2: two FMAs an instruction), so both operands stay in shared memory as they lie in global memory, rows of K
// padded by 16 bytes: a quarter warp reads eight consecutive rows without conflicts, and an operand needs no transposition.
//
// Products with few tiles share K out over a cluster of up to eight CTAs.  Each pushes its sums to the CTAs that own the rows
// (shared memory of the cluster), which add them in rank order: same result every time, no workspace.
//
// 2 rows, down product 2048 x 8192, weights cold: 705 -> 41 us against the tiles of twm_dense_simt.cuh, which copy element by element
// with nothing in flight; those stay for rows that are not on 16-byte boundaries.  More rows: twm_dense_f32tc.cuh.
#pragma once

#include "twm_dense_common.cuh"

namespace twm {
namespace dense {

constexpr int F32_ROWS = 8, F32_BK = 32, F32_LD = F32_BK + 4, F32_BN = 128, F32_THREADS = 256, F32_STAGES = 3, F32_MAX_SPLITS = 8;
constexpr int F32_STAGE_FLOATS = (F32_ROWS + F32_BN) * F32_LD;
constexpr size_t F32_SMEM_BYTES = sizeof(float) * (size_t)F32_STAGES * F32_STAGE_FLOATS;

struct GemmF32Args {
    const float *a, *w;
    float* c;
    int lda, ldw, ldc, M, N, K;     // gated: N output columns, 2 N weight rows
    int splits;
};

__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

template <int EPI>
__global__ void __launch_bounds__(F32_THREADS, 2)
gemm_f32_kernel(const GemmF32Args g)
{
    constexpr bool GATED = EPI == TWM_EPI_GELU_GLU;
    constexpr int BM = F32_ROWS, TN = F32_BN / 32, OUT = GATED ? F32_BN / 2 : F32_BN, STAGE = F32_STAGE_FLOATS;
    extern __shared__ __align__(16) float f32_smem[];
    pdl_launch_dependents();
    const int tid = threadIdx.x, lane = tid & 31;
    const int rank = blockIdx.x % g.splits, tile = blockIdx.x / g.splits;
    const int n0 = tile * OUT;
    const int k_tiles = (g.K + F32_BK - 1) / F32_BK, per = (k_tiles + g.splits - 1) / g.splits;
    const int k_first = min(k_tiles, rank * per), steps = min(k_tiles, k_first + per) - k_first;

    // 16-byte pieces of a stage: eight threads read 128 contiguous bytes of a row
    const int piece = (tid & 7) * 4, row0 = tid >> 3;
    auto load_w = [&](int step) {
        float* ws = f32_smem + (step % F32_STAGES) * STAGE + BM * F32_LD;
        const int k = (k_first + step) * F32_BK + piece, bytes = max(0, min(4, g.K - k)) * 4;
#pragma unroll
        for (int i = 0; i < TN; ++i) {
            const int r = row0 + i * 32, n = n0 + (GATED ? r % OUT : r);
            const bool in = n < g.N && bytes > 0;
            const float* src = g.w + (in ? (size_t)(GATED && r >= OUT ? g.N + n : n) * g.ldw + k : 0);
            ops::att_cp_async16(smem_u32(ws + r * F32_LD + piece), src, in ? bytes : 0);
        }
    };
    auto load_a = [&](int step) {
        float* as = f32_smem + (step % F32_STAGES) * STAGE;
        const int k = (k_first + step) * F32_BK + piece, bytes = max(0, min(4, g.K - k)) * 4;
        if (row0 >= BM) return;
        const bool in = row0 < g.M && bytes > 0;
        ops::att_cp_async16(smem_u32(as + row0 * F32_LD + piece), g.a + (in ? (size_t)row0 * g.lda + k : 0), in ? bytes : 0);
    };
    // weights are constants: the first stages of them are on their way before the preceding kernel has ended
#pragma unroll
    for (int s = 0; s < F32_STAGES - 1; ++s)
        if (s < steps) load_w(s);
    pdl_wait_prior_grids();
#pragma unroll
    for (int s = 0; s < F32_STAGES - 1; ++s) {
        if (s < steps) load_a(s);
        ops::att_cp_async_commit();
    }

    const int tr = lane & 7, tc = (tid >> 5) * 4 + (lane >> 3);     // row tr, weight rows tc + 32 j
    uint64_t acc[TN];
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[j] = 0;
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group %0;" ::"n"(F32_STAGES - 2) : "memory");
        __syncthreads();                                            // the stage is there, and the one before it has been used
        if (step + F32_STAGES - 1 < steps) { load_w(step + F32_STAGES - 1); load_a(step + F32_STAGES - 1); }
        ops::att_cp_async_commit();
        const float* as = f32_smem + (step % F32_STAGES) * STAGE + tr * F32_LD;
        const float* ws = f32_smem + (step % F32_STAGES) * STAGE + (BM + tc) * F32_LD;
#pragma unroll
        for (int k = 0; k < F32_BK; k += 4) {
            const ulonglong2 av = *reinterpret_cast<const ulonglong2*>(as + k);
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const ulonglong2 wv = *reinterpret_cast<const ulonglong2*>(ws + j * 32 * F32_LD + k);
                fma2(acc[j], av.x, wv.x);
                fma2(acc[j], av.y, wv.y);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    // every CTA of the cluster has used its stages; the sums go to the owners of their rows
    const int own = (BM + g.splits - 1) / g.splits;
    if (g.splits > 1) cluster_sync_all(); else __syncthreads();
    const int owner = g.splits > 1 ? tr / own : 0;
    float* to = f32_smem + ((size_t)rank * own + (tr - owner * own)) * F32_BN + tc;
    const uint32_t remote = g.splits > 1 ? mapa_shared(smem_u32(to), owner) : 0;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
        const float v = __uint_as_float((uint32_t)acc[j]) + __uint_as_float((uint32_t)(acc[j] >> 32));
        if (g.splits > 1) st_cluster_f32(remote + j * 32 * 4, v);
        else to[j * 32] = v;
    }
    if (g.splits > 1) cluster_sync_all(); else __syncthreads();
    for (int i = tid; i < own * OUT; i += F32_THREADS) {
        const int r = i / OUT, n = i - r * OUT, m = rank * own + r;
        if (m >= g.M || n0 + n >= g.N) continue;
        float v = 0.0f, up = 0.0f;
        for (int s = 0; s < g.splits; ++s) {
            v += f32_smem[((size_t)s * own + r) * F32_BN + n];
            if (GATED) up += f32_smem[((size_t)s * own + r) * F32_BN + OUT + n];
        }
        g.c[(size_t)m * g.ldc + n0 + n] = GATED ? gelu_tanh(v) * up : epilogue_value<EPI>(v);
    }
}

}  // namespace dense
}  // namespace twm
