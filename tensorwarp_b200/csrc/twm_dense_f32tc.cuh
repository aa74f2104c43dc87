// twm_dense_f32tc.cuh — C[M][N] = A[M][K] . W[N][K]^T of the 32-bit models on the tensor cores, with the error of an FP32 product.
//
// An FP32 number is the sum of three bfloat16 numbers: itself rounded to the nearest, what that leaves rounded to the nearest, and the
// rest (23 bits and two signs: nothing is left).  The last of them lies up to 2^-23 below the number, so operands are multiplied by 2^24
// first and the sums by 2^-48 at the end, both exactly: below 2^-110 the parts would run into bfloat16's smallest number (2^-133) and
// be cut (activations of 2^-120, K = 1024: errors of 1.6e-5 of the sum of absolute products without the factor, 2.7e-8 with it, 2.4e-7
// in FP32 FMAs).  A product of two is the sum of nine; the six largest are taken, the others are below 2^-24 of it, which is
// what an FP32 product rounds by (cut instead of rounded parts: 2^-21).  The tensor core multiplies them exactly, but cuts when it adds.  So the products of the leading parts (acc 0)
// and the other five (acc 1, 2^-8 smaller) have accumulators of their own, and both are taken out and added up in FP32
// registers every 64 K.
//
// Tile: 128 weight rows (the MMA's M) x up to 128 activation rows, 64 K a stage, two stages, one CTA to an SM, K shared by a
// cluster of up to eight.  Warps 0-7 take accumulators out (thread = weight row, every second chunk of 16 activation rows),
// 8-15 read FP32 rows from global memory, split them and write the six operands to shared memory, 16 issues the MMAs.  A stage moves
// 160 KB through shared memory at 80 rows.  What bounds it is the splitting, with the wait for its loads: gate/up of 70 rows, 64.2 us, without MMAs
// 59.5, without loads 52.4, without either 47.8, without splitting 41.
//
// A number that is not finite, or not below 2^104, has no such sum: its second part is not a number, nor is any sum that it enters.  The
// reading threads notice that, or a sum that has outgrown FP32 (from 2^80 on with the factors), and the cluster computes its tile
// with plain FP32 FMAs instead.
#pragma once

#include "twm_dense_f32.cuh"
#include "twm_dense_tcs.cuh"

namespace twm {
namespace dense {

constexpr int FX_BN = 128, FX_BK = 64, FX_MAX_ROWS = 128, FX_CORES = FX_BK / 8;
constexpr int FX_READERS = 256, FX_SPLITTERS = 256, FX_THREADS = FX_READERS + FX_SPLITTERS + 32, FX_LD = FX_BN + 4;
// An operand part: [row][64 K], 128 bytes a row, its 16-byte pieces in the order of the 128-byte swizzle: the eight threads on a row write
// one line, and the MMA reads whole lines.  (K cores of 8 x 16 bytes, 16 bytes apart so that the writes met no bank twice, lay across
// the lines: gate/up of a 70-row prompt, 16384 x 2048, 72.4 us against 66.6; out and down 35.9 against 29.8 on average.)
__host__ __device__ constexpr int fx_part_bytes(int rows) { return rows * FX_BK * 2; }
__host__ __device__ constexpr int fx_stage_bytes(int bm) { return 3 * (fx_part_bytes(FX_BN) + fx_part_bytes(bm)); }
inline size_t fx_smem_bytes(int bm) { return std::max(2 * fx_stage_bytes(bm), bm * FX_LD * 4) + 1024; }

constexpr float FX_SCALE = 16777216.0f, FX_UNSCALE = 1.0f / (FX_SCALE * FX_SCALE);     // 2^24 and 2^-48

struct GemmFxArgs {
    const float *a, *w;
    float* c;
    int lda, ldw, ldc, M, N, K;     // gated: N output columns, 2 N weight rows
    int m_tiles, bm, splits;        // bm: activation rows a tile, a multiple of 16
};

// Rows first ... (count of them) of a tile with FP32 FMAs: a warp takes two rows x four weight rows, its lanes along K.  70 rows, 2048 x
// 8192, one NaN: 6 714 us with a thread along K for each four results, 330 us this way (the plain tiles of twm_dense_simt.cuh: 573); 1024 rows: 71 204 and 3 031.
template <int EPI>
__device__ __forceinline__ void fx_plain(const GemmFxArgs g, int first, int count, int n0)
{
    constexpr bool GATED = EPI == TWM_EPI_GELU_GLU;
    constexpr int COLS = GATED ? 2 : 4, ITEMS = FX_BN / 4;
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int i = threadIdx.x >> 5; i < (count + 1) / 2 * ITEMS; i += FX_THREADS / 32) {
        const int m = first + i / ITEMS * 2, n = n0 + i % ITEMS * COLS;
        if (n >= g.N) continue;
        const float *a0 = g.a + (size_t)m * g.lda, *a1 = a0 + (m + 1 < first + count ? g.lda : 0), *w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = g.w + (size_t)(min(n + j % COLS, g.N - 1) + (GATED && j >= COLS ? g.N : 0)) * g.ldw;
        float s[8] = {};
#pragma unroll 2
        for (int k = lane * 4; k < g.K; k += 128) {
            auto four = [&](const float* p) {
                if (k + 4 <= g.K) return *reinterpret_cast<const float4*>(p + k);
                return make_float4(p[k], k + 1 < g.K ? p[k + 1] : 0.f, k + 2 < g.K ? p[k + 2] : 0.f, 0.f);
            };
            const float4 x = four(a0), y = four(a1);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float4 v = four(w[j]);
                s[j] = fmaf(x.w, v.w, fmaf(x.z, v.z, fmaf(x.y, v.y, fmaf(x.x, v.x, s[j]))));
                s[4 + j] = fmaf(y.w, v.w, fmaf(y.z, v.z, fmaf(y.y, v.y, fmaf(y.x, v.x, s[4 + j]))));
            }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) s[j] = ops::warp_sum(s[j]);
        if (lane == 0) {
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int j = 0; j < COLS; ++j)
                    if (m + r < first + count && n + j < g.N)
                        g.c[(size_t)(m + r) * g.ldc + n + j] = GATED ? gelu_tanh(s[4 * r + j]) * s[4 * r + 2 + j] : s[4 * r + j];
        }
    }
}

template <int EPI>
__global__ void __launch_bounds__(FX_THREADS, 1)
gemm_f32tc_kernel(const GemmFxArgs g)
{
    constexpr bool GATED = EPI == TWM_EPI_GELU_GLU;
    constexpr int OUT = GATED ? FX_BN / 2 : FX_BN;
    extern __shared__ uint8_t fx_smem_raw[];
    uint8_t* fx_smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(fx_smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t full[2], empty[2], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_s;
    __shared__ int abort_s;
    __shared__ __align__(16) float odd_s[4];         // [0]: not zero where a number has no split or a sum is not finite
    volatile int* abort_flag = &abort_s;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = blockIdx.x % g.splits, tile = blockIdx.x / g.splits;
    const int m0 = tile % g.m_tiles * g.bm, n0 = tile / g.m_tiles * OUT, rows = min(g.bm, g.M - m0);
    const int k_tiles = (g.K + FX_BK - 1) / FX_BK;
    const int k_first = (int)((long)rank * k_tiles / g.splits), steps = (int)((long)(rank + 1) * k_tiles / g.splits) - k_first;
    const int stage_bytes = fx_stage_bytes(g.bm), w_part = fx_part_bytes(FX_BN), a_part = fx_part_bytes(g.bm);

    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&full[i], FX_SPLITTERS / 32); mbar_init(&empty[i], 1);
            mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], FX_READERS / 32);
        }
        abort_s = 0;
        odd_s[0] = odd_s[1] = odd_s[2] = odd_s[3] = 0.0f;
        mbar_fence_init();
    }
    if (warp == FX_THREADS / 32 - 1) {
        tc::tmem_alloc(&tmem_s, 512);
        tc::tc_fence_before();
    }
    __syncthreads();
    tc::tc_fence_after();
    pdl_launch_dependents();
    cluster_started();
    const uint32_t tmem = tmem_s;
    float acc[64];                                    // readers: sums of chunks 2 i + (warp >> 2)

    if (warp == FX_THREADS / 32 - 1) {
        // ------------------------------------------------------------ MMAs --
        if (elect_one()) {
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(g.bm >> 3) << 17) | ((uint32_t)(FX_BN >> 4) << 24);
            bool ok = true;
            for (int t = 0; t < steps && ok; ++t) {
                const int s = t & 1;
                if (!mbar_wait_bounded(&full[s], (t >> 1) & 1, abort_flag)) { ok = false; break; }
                if (t >= 2 && !mbar_wait_bounded(&acc_empty[s], ((t >> 1) - 1) & 1, abort_flag)) { ok = false; break; }
                tc::tc_fence_after();
                const uint32_t base = smem_u32(fx_smem + s * stage_bytes);
                // (part of W, part of A): the leading parts into accumulator 0, the five next smaller products into 1
                auto product = [&](int wp, int ap, uint32_t d, bool first) {
                    uint64_t wd = sw128_desc(base + wp * w_part), ad = sw128_desc(base + 3 * w_part + ap * a_part);
#pragma unroll
                    for (int h = 0; h < FX_BK / 16; ++h) {               // 16 K = 32 bytes further along the swizzled rows
                        tcw::mma_ss(d, wd, ad, idesc, first && h == 0 ? 0u : 1u);
                        wd += 2;
                        ad += 2;
                    }
                };
                const uint32_t d = tmem + s * 256;
                product(0, 0, d, true);
                product(0, 2, d + 128, true);
                product(2, 0, d + 128, false);
                product(1, 1, d + 128, false);
                product(0, 1, d + 128, false);
                product(1, 0, d + 128, false);
                tc::tc_commit(&empty[s]);
                tc::tc_commit(&acc_full[s]);
            }
        }
        __syncwarp();
    } else if (warp >= FX_READERS / 32) {
        // ------------------------------------------------------- splitting --
        const int st = tid - FX_READERS, row0 = st >> 3, core = st & 7;      // rows row0 + 32 j, eight K each
        float4 x[8][2];                               // 0-3: weight rows, 4-7: activation rows
        const int k_lane = k_first * FX_BK + core * 8;
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j][0] = x[j][1] = make_float4(0.f, 0.f, 0.f, 0.f);
        auto load = [&](int j, int t) {               // rows that are not there stay zero
            const float* p;
            if (j < 4) {
                const int n = n0 + row0 + (GATED ? j & 1 : j) * 32;
                if (n >= g.N) return;
                p = g.w + (size_t)(GATED && j >= 2 ? g.N + n : n) * g.ldw;
            } else {
                const int r = row0 + (j - 4) * 32;
                if (r >= rows) return;
                p = g.a + (size_t)(m0 + r) * g.lda;
            }
            p += k_lane + t * FX_BK;
            const int left = g.K - k_lane - t * FX_BK;
            if (left >= 8) {
                x[j][0] = *reinterpret_cast<const float4*>(p);
                x[j][1] = *reinterpret_cast<const float4*>(p + 4);
                return;
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                x[j][h] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (4 * h + 4 <= left) {
                    x[j][h] = *reinterpret_cast<const float4*>(p + 4 * h);
                } else {
                    if (4 * h < left) x[j][h].x = p[4 * h];
                    if (4 * h + 1 < left) x[j][h].y = p[4 * h + 1];
                    if (4 * h + 2 < left) x[j][h].z = p[4 * h + 2];
                }
            }
        };
        auto split = [&](int j, uint8_t* dst, int part_bytes) {
            const float v[8] = {x[j][0].x, x[j][0].y, x[j][0].z, x[j][0].w, x[j][1].x, x[j][1].y, x[j][1].z, x[j][1].w};
            uint32_t o[3][4];
#pragma unroll
            for (int i = 0; i < 8; i += 2) {
                float f[2] = {v[i] * FX_SCALE, v[i + 1] * FX_SCALE};
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    const __nv_bfloat162 b = __floats2bfloat162_rn(f[0], f[1]);
                    o[q][i >> 1] = *reinterpret_cast<const uint32_t*>(&b);
                    if (q == 2) break;
                    f[0] -= __uint_as_float(o[q][i >> 1] << 16);
                    f[1] -= __uint_as_float(o[q][i >> 1] & 0xffff0000u);
                }
            }
#pragma unroll
            for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4*>(dst + q * part_bytes) = make_uint4(o[q][0], o[q][1], o[q][2], o[q][3]);
        };
        // weights are constants: the first ones are on their way before the preceding kernel has ended
#pragma unroll
        for (int j = 0; j < 4; ++j) if (steps > 0) load(j, 0);
        pdl_wait_prior_grids();
#pragma unroll
        for (int j = 4; j < 8; ++j) if (steps > 0) load(j, 0);
        for (int t = 0; t < steps; ++t) {
            const int s = t & 1;
            if (t >= 2 && !tc::wait_uniform(&empty[s], ((t >> 1) - 1) & 1, abort_flag)) break;
            uint8_t* base = fx_smem + s * stage_bytes;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int r = row0 + (j & 3) * 32;
                uint8_t* piece = base + r * 128 + ((core ^ (r & 7)) << 4);
                if (j < 4) split(j, piece, w_part);
                else if (r < g.bm) split(j, piece + 3 * w_part, a_part);
                if (t + 1 < steps) load(j, t + 1);
            }
            // written through the generic proxy, read by the tensor core through the async proxy
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
        }
    } else {
        // -------------------------------------------------------- read-back --
#pragma unroll
        for (int i = 0; i < 64; ++i) acc[i] = 0.0f;
        const uint32_t at = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        for (int t = 0; t < steps; ++t) {
            const int s = t & 1;
            if (!tc::wait_uniform(&acc_full[s], (t >> 1) & 1, abort_flag)) break;
            tc::tc_fence_after();
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int c0 = (2 * i + (warp >> 2)) * 16;
                if (c0 < g.bm) {                      // warp-uniform
                    uint32_t d0[16], d1[16];
                    tc::tmem_ld<16>(at + s * 256 + c0, d0);
                    tc::tmem_ld<16>(at + s * 256 + 128 + c0, d1);
                    tc::tmem_wait_ld();
#pragma unroll
                    for (int e = 0; e < 16; ++e) acc[i * 16 + e] += __uint_as_float(d0[e]) + __uint_as_float(d1[e]);
                }
            }
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[s]);
        }
        bool fine = true;
#pragma unroll
        for (int i = 0; i < 64; ++i) fine = fine && fabsf(acc[i]) < INFINITY;
        if (!fine) odd_s[0] = 1.0f;
    }
    __syncthreads();                                  // every MMA has run: the sums go where the stages were
    float* sums = reinterpret_cast<float*>(fx_smem);  // [activation row][FX_LD]
    if (warp < FX_READERS / 32) {
        const int n = (warp & 3) * 32 + lane;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int c0 = (2 * i + (warp >> 2)) * 16;
            if (c0 < g.bm) {
#pragma unroll
                for (int e = 0; e < 16; ++e) sums[(c0 + e) * FX_LD + n] = acc[i * 16 + e];
            }
        }
    }
    const bool all_ok = cluster_meet(abort_flag);
    const int own = (rows + g.splits - 1) / g.splits, first = rank * own;
    if (!all_ok) {
        // a wait ran out: nothing is stored, the error word is set
    } else if (cluster_sum4(odd_s, g.splits).x != 0.0f) {    // the same in every CTA: nobody reads the sums
        fx_plain<EPI>(g, m0 + first, min(own, rows - first), n0);
    } else {
        for (int i = tid; i < own * (OUT / 4); i += FX_THREADS) {
            const int r = i / (OUT / 4), col = (i - r * (OUT / 4)) * 4, m = first + r;
            if (m >= rows || n0 + col >= g.N) continue;
            const float4 x = cluster_sum4(sums + m * FX_LD + col, g.splits);
            float v[4] = {x.x * FX_UNSCALE, x.y * FX_UNSCALE, x.z * FX_UNSCALE, x.w * FX_UNSCALE};
            if (GATED) {
                const float4 z = cluster_sum4(sums + m * FX_LD + OUT + col, g.splits);
                const float u[4] = {z.x * FX_UNSCALE, z.y * FX_UNSCALE, z.z * FX_UNSCALE, z.w * FX_UNSCALE};
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] = gelu_tanh(v[j]) * u[j];
            }
            tc_store4<TWM_EPI_STORE_F32>(g.c, (size_t)(m0 + m) * g.ldc, n0 + col, g.N, v);
        }
    }
    cluster_sync_all();                               // nobody leaves while its sums may still be read
    if (warp == FX_THREADS / 32 - 1) {
        tc::tc_fence_after();
        tc::tmem_dealloc(tmem, 512);
    }
}

}  // namespace dense
}  // namespace twm
