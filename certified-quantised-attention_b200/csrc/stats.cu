// Per-step telemetry of a finished layer step in one launch: what the stats dict needs beyond the certificate
// (promoted blocks, mass sums, error and norm maxima), written behind the certificate so that one copy brings both to
// the host.  (As torch reductions these were a dozen launches with a synchronisation each, 700 of the 800 us of a
// step with stats at 8192 tokens.)
//
// Words of `out`: [H] blocks not in the FP16-key mask (int) | [H] sum of the mass fractions (float) | [KV] largest
// eta_b of the whole array (float) | [KV] largest nu_b of the active blocks (float) | [CQA_STATS_PARTS] blocks that
// any head reads from Tier 2, by part (int).
#include "common.cuh"

namespace cqa {

constexpr int ST_THREADS = 256;

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

__global__ void __launch_bounds__(ST_THREADS) step_stats_kernel(cqa_cache c, cqa_workspace ws, int H, int nq, int nact, int32_t *out)
{
    __shared__ int s_i[ST_THREADS / 32];
    __shared__ float s_f[ST_THREADS / 32];
    const int x = blockIdx.x, tid = threadIdx.x;
    const auto add_i = [](int a, int b) { return a + b; };
    const auto add_f = [](float a, float b) { return a + b; };
    const auto max_f = [](float a, float b) { return fmaxf(a, b); };
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
    } else if (x < H + c.kv_heads) {
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
            out[2 * H + c.kv_heads + kv] = __float_as_int(nu);
        }
    } else {
        const int part = x - H - c.kv_heads, per = (nq + CQA_STATS_PARTS - 1) / CQA_STATS_PARTS;
        int n = 0;
        for (int b = part * per + tid; b < min(nq, (part + 1) * per); b += ST_THREADS) {
            int any = 0;
#pragma unroll 8
            for (int h = 0; h < H; ++h) any |= ws.value_mask[(long)h * ws.ld + b];
            n += any != 0 ? 1 : 0;
        }
        n = cta_reduce(n, s_i, add_i);
        if (tid == 0) out[2 * H + 2 * c.kv_heads + part] = n;
    }
}

}  // namespace cqa

using namespace cqa;

extern "C" int cqa_step_stats(const cqa_cache *c, const cqa_workspace *ws, int64_t nq, int64_t nact, void *out, void *stream)
{
    if (!c || !ws || !out || !ws->topk_mask || !ws->value_mask || !ws->mass_frac) { set_error("cqa_step_stats: NULL pointer"); return CQA_ERR_INVALID; }
    if (nq < 0 || nact < nq || nact > ws->ld || nact > c->max_blocks || c->kv_heads <= 0 || c->gqa_group <= 0) {
        set_error("cqa_step_stats: sizes out of range");
        return CQA_ERR_INVALID;
    }
    const int H = c->kv_heads * c->gqa_group;
    step_stats_kernel<<<H + c->kv_heads + CQA_STATS_PARTS, ST_THREADS, 0, (cudaStream_t)stream>>>(*c, *ws, H, (int)nq, (int)nact,
                                                                                                 static_cast<int32_t *>(out));
    note_launch();
    return check_launch("step_stats_kernel");
}
