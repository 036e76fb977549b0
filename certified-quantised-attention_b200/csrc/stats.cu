// Per-step telemetry of a finished layer step: every sum, mean, minimum and maximum that the stats dict needs, reduced
// on the device by one launch whose last CTA writes a few dozen numbers into the caller's (pinned) memory.  (As torch
// reductions these were a dozen launches with a synchronisation each, 700 of the 800 us of a step with stats at 8192
// tokens; with the certificate copied and its columns summed by the interpreter 155 us were left.)
//
// Scratch words: [H] blocks not in the FP16-key mask (int) | [H] sum of the mass fractions (float) | [KV] largest eta_b of
// the whole array (float) | [KV] largest nu_b of the active blocks (float) | [STAT_PARTS] blocks that any head reads from
// Tier 2, by part (int) | ticket.
#include <stddef.h>

#include "common.cuh"

namespace cqa {

constexpr int ST_THREADS = 256;
constexpr int STAT_PARTS = 16;

template <typename T, typename F>
__device__ __forceinline__ T cta_reduce(T v, T *s, F op)
{
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) v = op(v, __shfl_xor_sync(FULL, v, o));
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
    __syncthreads();
    v = s[threadIdx.x & (ST_THREADS / 32 - 1)];
#pragma unroll
    for (int o = ST_THREADS / 64; o >= 1; o >>= 1) v = op(v, __shfl_xor_sync(FULL, v, o));
    return v;
}

// What the summary holds, by position: a reduction over the heads' certificate fields, or over a row of the scratch words.
enum StatKind : unsigned char { S_INT_SUM, S_INT_MIN, S_INT_MAX, S_F_SUM, S_F_MAX, S_GAP_SUM, S_GAP_MIN, S_EKEY_SUM, S_EKEY_MAX, S_FLAG,
                                S_SKIPPED, S_RHO_SUM, S_RHO_MAX, S_ETA, S_NU, S_UNION };
struct StatItem {
    StatKind kind;
    unsigned short offset;
};
#define F_(name) (unsigned short)offsetof(cqa_head_cert, name)
__constant__ StatItem g_items[CQA_SUMMARY_ITEMS] = {
    {S_FLAG, 2}, {S_INT_SUM, F_(consistency_violation)}, {S_INT_SUM, F_(boundary_triggered)}, {S_INT_SUM, F_(rung1_triggered)},
    {S_INT_SUM, F_(value_promoted_blocks)}, {S_INT_SUM, F_(dense)}, {S_INT_SUM, F_(exploration_blocks)},
    {S_INT_SUM, F_(ranking_disagree_r1)}, {S_INT_SUM, F_(ranking_disagree_r3)},
    {S_INT_SUM, F_(k_star)}, {S_INT_MIN, F_(k_star)}, {S_INT_MAX, F_(k_star)},
    {S_F_SUM, F_(delta)}, {S_F_SUM, F_(e_val)}, {S_F_MAX, F_(e_val)}, {S_F_SUM, F_(e_pre)}, {S_F_MAX, F_(e_pre)},
    {S_F_SUM, F_(tau_actual)}, {S_F_SUM, F_(tail_mass)}, {S_F_MAX, F_(tail_mass)}, {S_F_SUM, F_(int8_top1)}, {S_F_SUM, F_(fp16_top1)},
    {S_GAP_SUM, 0}, {S_GAP_MIN, 0}, {S_EKEY_SUM, 0}, {S_EKEY_MAX, 0},
    {S_SKIPPED, 0}, {S_RHO_SUM, 0}, {S_RHO_MAX, 0}, {S_ETA, 0}, {S_NU, 0}, {S_UNION, 0},
};
#undef F_

__device__ __forceinline__ double warp_reduce_item(const StatItem it, const cqa_workspace &ws, int H, int KV, const int32_t *w)
{
    const int lane = threadIdx.x & 31;
    const bool is_max = it.kind == S_INT_MAX || it.kind == S_F_MAX || it.kind == S_EKEY_MAX || it.kind == S_RHO_MAX || it.kind == S_ETA || it.kind == S_NU;
    const bool is_min = it.kind == S_INT_MIN || it.kind == S_GAP_MIN;
    double acc = is_max ? -INFINITY : (is_min ? INFINITY : 0.0);
    const auto take = [&](double v) { acc = is_max ? fmax(acc, v) : (is_min ? fmin(acc, v) : acc + v); };
    if (it.kind < S_FLAG) {
        for (int h = lane; h < H; h += 32) {
            const char *ct = reinterpret_cast<const char *>(ws.cert + h);
            if (it.kind <= S_INT_MAX) {
                take((double)*reinterpret_cast<const int32_t *>(ct + it.offset));
            } else if (it.kind <= S_F_MAX) {
                take((double)*reinterpret_cast<const float *>(ct + it.offset));
            } else if (it.kind <= S_GAP_MIN) {
                take((double)__fsub_rn(ws.cert[h].fp16_top1, ws.cert[h].fp16_top2));
            } else {
                const double e = exp(2.0 * (double)ws.cert[h].delta);      // without the layer's largest value norm
                take(2.0 * e * (double)ws.cert[h].tail_mass * (e - 1.0));
            }
        }
    } else if (it.kind == S_FLAG) {
        if (lane == 0) acc = (double)ws.any_flags[it.offset];
    } else {
        const int first = it.kind == S_SKIPPED ? 0 : it.kind <= S_RHO_MAX ? H : it.kind == S_ETA ? 2 * H : it.kind == S_NU ? 2 * H + KV : 2 * (H + KV);
        const int count = it.kind <= S_RHO_MAX ? H : it.kind <= S_NU ? KV : STAT_PARTS;
        const bool integer = it.kind == S_SKIPPED || it.kind == S_UNION;
        for (int i = lane; i < count; i += 32) {
            const int v = __ldcg(w + first + i);
            take(integer ? (double)v : (double)__int_as_float(v));
        }
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        const double x = __shfl_xor_sync(FULL, acc, o);
        acc = is_max ? fmax(acc, x) : (is_min ? fmin(acc, x) : acc + x);
    }
    return acc;
}

__global__ void __launch_bounds__(ST_THREADS) step_stats_kernel(const __grid_constant__ cqa_cache c, const __grid_constant__ cqa_workspace ws,
                                                               int H, int nq, int nact, int32_t *out, double *summary)
{
    __shared__ int s_i[ST_THREADS / 32];
    __shared__ float s_f[ST_THREADS / 32];
    __shared__ int s_last;
    const int x = blockIdx.x, tid = threadIdx.x, KV = c.kv_heads;
    const auto add_i = [](int a, int b) { return a + b; };
    const auto add_f = [](float a, float b) { return a + b; };
    const auto max_f = [](float a, float b) { return fmaxf(a, b); };
    grid_dependency_wait();
    if (x < H) {
        const uint8_t *mask = ws.topk_mask + (long)x * ws.ld;
        const float *frac = ws.mass_frac + (long)x * ws.ld;
        int skipped = 0;
        float rho = 0.0f;
#pragma unroll 4
        for (int b = tid; b < nact; b += ST_THREADS) skipped += mask[b] == 0 ? 1 : 0;
#pragma unroll 4
        for (int b = tid; b < nq; b += ST_THREADS) rho += frac[b];
        skipped = cta_reduce(skipped, s_i, add_i);
        rho = cta_reduce(rho, s_f, add_f);
        if (tid == 0) {
            out[x] = skipped;
            out[H + x] = __float_as_int(rho);
        }
    } else if (x < H + KV) {
        const int kv = x - H;
        const long row = (long)kv * c.max_blocks;
        float eta = 0.0f, nu = 0.0f;
        if (c.values_int4_errors) {
#pragma unroll 4
            for (int b = tid; b < (int)c.max_blocks; b += ST_THREADS) eta = fmaxf(eta, c.values_int4_errors[row + b]);
        }
        if (c.values_norm_max) {
#pragma unroll 4
            for (int b = tid; b < nact; b += ST_THREADS) nu = fmaxf(nu, c.values_norm_max[row + b]);
        }
        eta = cta_reduce(eta, s_f, max_f);
        __syncthreads();
        nu = cta_reduce(nu, s_f, max_f);
        if (tid == 0) {
            out[2 * H + kv] = __float_as_int(eta);
            out[2 * H + KV + kv] = __float_as_int(nu);
        }
    } else {
        const int part = x - H - KV, per = (nq + STAT_PARTS - 1) / STAT_PARTS;
        int n = 0;
        for (int b = part * per + tid; b < min(nq, (part + 1) * per); b += ST_THREADS) {
            int any = 0;
#pragma unroll 8
            for (int h = 0; h < H; ++h) any |= ws.value_mask[(long)h * ws.ld + b];
            n += any != 0 ? 1 : 0;
        }
        n = cta_reduce(n, s_i, add_i);
        if (tid == 0) out[2 * (H + KV) + part] = n;
    }
    // the last CTA reduces the rows and the certificate
    if (tid == 0) {
        __threadfence();
        int32_t *ticket = out + 2 * (H + KV) + STAT_PARTS;
        const int t = atomicAdd(ticket, 1);
        s_last = t == (int)gridDim.x - 1;
        if (s_last) { *ticket = 0; __threadfence(); }
    }
    __syncthreads();
    if (!s_last) return;
    for (int i = tid >> 5; i < CQA_SUMMARY_ITEMS; i += ST_THREADS / 32) {
        const double v = warp_reduce_item(g_items[i], ws, H, KV, out);
        if ((tid & 31) == 0) summary[i] = v;
    }
}

}  // namespace cqa

using namespace cqa;

extern "C" int cqa_step_stats(const cqa_cache *c, const cqa_workspace *ws, int64_t nq, int64_t nact, void *scratch,
                              double *summary_host, void *stream)
{
    if (!c || !ws || !scratch || !summary_host || !ws->topk_mask || !ws->value_mask || !ws->mass_frac || !ws->cert || !ws->any_flags) {
        set_error("cqa_step_stats: NULL pointer");
        return CQA_ERR_INVALID;
    }
    if (nq < 0 || nact < nq || nact > ws->ld || nact > c->max_blocks || c->kv_heads <= 0 || c->gqa_group <= 0) {
        set_error("cqa_step_stats: sizes out of range");
        return CQA_ERR_INVALID;
    }
    const int H = c->kv_heads * c->gqa_group;
    cudaStream_t st = (cudaStream_t)stream;
    void *mapped = nullptr;
    int rc = check_cuda(cudaHostGetDevicePointer(&mapped, summary_host, 0), "cqa_step_stats: summary_host must be pinned memory");
    if (rc) return rc;
    rc = check_cuda(launch_chained(step_stats_kernel, dim3((unsigned)(H + c->kv_heads + STAT_PARTS)), dim3(ST_THREADS), 0, st, true, *c, *ws,
                                   H, (int)nq, (int)nact, static_cast<int32_t *>(scratch), static_cast<double *>(mapped)),
                    "step_stats_kernel");
    if (rc) return rc;
    return check_cuda(cudaStreamSynchronize(st), "cudaStreamSynchronize");
}
