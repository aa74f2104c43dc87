// twm_dense_attn_f32.cuh — windowed sigmoid attention of a portion of a prompt in FP32, value heads of up to 128 columns.
//
// CTA = 8 or 32 queries of one head, a warp takes one or four.  Keys and values come 32 at a time into shared memory (cp.async, three
// tiles), where a lane first takes a key (rows are padded so that eight lanes read distinct banks), then four value columns.
// A sum is taken in the order of attn_simt_kernel, one query per CTA, whose bits it gives; that one reads every key
// and value from the L2 cache for every query: 70 queries, 16 heads of 128, in a prompt step: 27 us, 17 this way.
#pragma once

#include "twm_dense_simt.cuh"

namespace twm {
namespace dense {

constexpr int AF_WARPS = 8, AF_THREADS = AF_WARPS * 32, AF_KEYS = 32, AF_TILES = 3;
__host__ inline size_t attn_f32_smem_bytes(int dim_pad, int vdim_pad, int nq) {
    return sizeof(float) * ((size_t)AF_WARPS * nq * dim_pad + AF_TILES * (size_t)AF_KEYS * (dim_pad + 4 + vdim_pad));
}

template <int NQ>
__global__ void __launch_bounds__(AF_THREADS)
attn_f32_kernel(const AttnArgs<float> g)
{
    pdl_launch_dependents();
    extern __shared__ __align__(16) float af_smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ld = g.dim_pad + 4;
    float* qs = af_smem;                                   // [8 NQ][dim_pad]
    float* ks = qs + AF_WARPS * NQ * g.dim_pad;            // [tiles][32][ld]
    float* vs = ks + AF_TILES * AF_KEYS * ld;              // [tiles][32][vdim_pad]
    const int r0 = blockIdx.x * AF_WARPS * NQ, h = blockIdx.y, kvh = h / (g.heads / g.kv_heads);
    g.prefetch_bias(h, r0, AF_WARPS * NQ);
    pdl_wait_prior_grids();
    const int pos0 = g.meta[0], kd = g.kv_heads * g.dim_pad, vd = g.kv_heads * g.vdim_pad;
    const float* kc = g.k_cache + (size_t)g.meta[1] * g.capacity * kd + kvh * g.dim_pad;
    const float* vc = g.v_cache + (size_t)g.meta[1] * g.capacity * vd + kvh * g.vdim_pad;
    const float* bias = g.bias_table != nullptr ? g.bias_table + (size_t)h * g.bias_len : nullptr;
    const int p0 = pos0 + r0, p1 = pos0 + min(g.rows, r0 + AF_WARPS * NQ) - 1;
    int sinks, lo;
    visible_range(p0, g.window, g.keep_first, sinks, lo);
    const int total = sinks + (p1 - lo + 1);               // keys that some query of the CTA sees, and those between
    auto key_of = [&](int t) { return t < sinks ? t : lo + (t - sinks); };
    auto load = [&](int t0, int buf) {
        const int kp = g.dim_pad / 4, vp = g.vdim_pad / 4;
        for (int i = tid; i < AF_KEYS * kp; i += AF_THREADS) {
            const int r = i / kp, c = (i - r * kp) * 4;
            if (t0 + r < total) ops::att_cp_async16(smem_u32(ks + (buf * AF_KEYS + r) * ld + c), kc + (size_t)key_of(t0 + r) * kd + c, 16);
        }
        for (int i = tid; i < AF_KEYS * vp; i += AF_THREADS) {
            const int r = i / vp, c = (i - r * vp) * 4;
            if (t0 + r < total) ops::att_cp_async16(smem_u32(vs + (buf * AF_KEYS + r) * g.vdim_pad + c), vc + (size_t)key_of(t0 + r) * vd + c, 16);
        }
    };
#pragma unroll
    for (int i = 0; i < AF_TILES - 1; ++i) {
        load(i * AF_KEYS, i);
        ops::att_cp_async_commit();
    }
    for (int i = tid; i < AF_WARPS * NQ * (g.dim_pad / 4); i += AF_THREADS) {
        const int r = i / (g.dim_pad / 4), c = (i - r * (g.dim_pad / 4)) * 4;
        *reinterpret_cast<float4*>(qs + r * g.dim_pad + c) =
            r0 + r < g.rows ? *reinterpret_cast<const float4*>(g.proj + (size_t)(r0 + r) * g.ld + h * g.dim_pad + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const float* qw = qs + warp * NQ * g.dim_pad;          // this warp's queries
    const int first = r0 + warp * NQ, col = lane * 4;
    float4 acc[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) acc[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int t0 = 0, buf = 0; t0 < total; t0 += AF_KEYS, buf = buf + 1 == AF_TILES ? 0 : buf + 1) {
        asm volatile("cp.async.wait_group %0;" ::"n"(AF_TILES - 2) : "memory");
        __syncthreads();                                   // the tile is there, and the one before has been used
        load(t0 + (AF_TILES - 1) * AF_KEYS, buf == 0 ? AF_TILES - 1 : buf - 1);
        ops::att_cp_async_commit();
        const float4* kr = reinterpret_cast<const float4*>(ks + (buf * AF_KEYS + lane) * ld);
        const int t = t0 + lane, key = key_of(t);
        float s[NQ], w[NQ];
        unsigned seen[NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const int p = pos0 + first + q;
            seen[q] = __ballot_sync(0xffffffffu, t < total && first + q < g.rows && key <= p && (p - key < g.window || key < g.keep_first));
            s[q] = 0.0f;
        }
#pragma unroll 4
        for (int d = 0; d < g.dim_pad / 4; ++d) {
            const float4 k = t < total ? kr[d] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const float4 v = *reinterpret_cast<const float4*>(qw + q * g.dim_pad + d * 4);
                s[q] = fmaf(k.w, v.w, fmaf(k.z, v.z, fmaf(k.y, v.y, fmaf(k.x, v.x, s[q]))));
            }
        }
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const bool mine = (seen[q] >> lane) & 1;
            const float b = mine && bias != nullptr ? __ldg(bias + (pos0 + first + q - key)) : 0.0f;
            w[q] = mine ? sigmoid_f32(fmaf(s[q], g.scale, b)) : 0.0f;
        }
        const float* v0 = vs + buf * AF_KEYS * g.vdim_pad + col;
#pragma unroll 4
        for (int tt = 0; tt < AF_KEYS; ++tt) {
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (t0 + tt < total && col < g.vdim_pad) v = *reinterpret_cast<const float4*>(v0 + tt * g.vdim_pad);
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const float wt = __shfl_sync(0xffffffffu, w[q], tt);
                if ((seen[q] >> tt) & 1) {                 // an unseen key's values may be anything
                    acc[q].x = fmaf(wt, v.x, acc[q].x); acc[q].y = fmaf(wt, v.y, acc[q].y);
                    acc[q].z = fmaf(wt, v.z, acc[q].z); acc[q].w = fmaf(wt, v.w, acc[q].w);
                }
            }
        }
    }
    if (col >= g.vdim_pad) return;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const int r = first + q;
        if (r >= g.rows) break;
        float4 o = acc[q];
        if (g.gate_off >= 0) {
            const float4 z = *reinterpret_cast<const float4*>(g.proj + (size_t)r * g.ld + g.gate_off + h * g.vdim_pad + col);
            o.x *= sigmoid_f32(z.x); o.y *= sigmoid_f32(z.y); o.z *= sigmoid_f32(z.z); o.w *= sigmoid_f32(z.w);
        }
        *reinterpret_cast<float4*>(g.out + (size_t)r * g.heads * g.vdim_pad + h * g.vdim_pad + col) = o;
    }
}

}  // namespace dense
}  // namespace twm
