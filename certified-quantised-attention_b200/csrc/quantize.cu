// Block quantisers: INT8 per-channel keys, INT4 per-token-per-group values,
// error annotations, and the fused append-and-quantise step.
//
// One CTA of 128 threads works on one (kv head, 16-token block).  Keys: thread c
// owns channel c over the 16 tokens.  Values: thread (t, g) owns group g of
// token t (16 channels).  All arithmetic that lands in stored bytes is
// elementwise IEEE; the error norms use the canonical 16-lane dot order.
#include <cstring>
#include <type_traits>

#include "common.cuh"

namespace cqa {

struct BlockQuantSmem {
    float scale[D];
    float tok_err[BS];
    float tok_vnorm[BS];
};

// Butterfly over the 16 lane-partials of one token held by 8 consecutive
// threads (thread g holds partials 2g and 2g+1).
__device__ __forceinline__ float group8_sum(float pa, float pb)
{
    pa = __fadd_rn(pa, __shfl_xor_sync(FULL, pa, 4));
    pb = __fadd_rn(pb, __shfl_xor_sync(FULL, pb, 4));
    pa = __fadd_rn(pa, __shfl_xor_sync(FULL, pa, 2));
    pb = __fadd_rn(pb, __shfl_xor_sync(FULL, pb, 2));
    pa = __fadd_rn(pa, __shfl_xor_sync(FULL, pa, 1));
    pb = __fadd_rn(pb, __shfl_xor_sync(FULL, pb, 1));
    return __fadd_rn(pa, pb);
}

__device__ __forceinline__ float sumsq16(const float (&x)[16], float &pa, float &pb)
{
    float a[8], b[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) { a[i] = x[i]; b[i] = x[i + 8]; }
    pa = chain8(a, a);
    pb = chain8(b, b);
    return 0.0f;
}

// INT4 quantisation of one (token, group): x[16] -> codes packed in 8 bytes,
// scale, zero, and the group's contribution to |x - deq|^2 (two lane partials).
__device__ __forceinline__ void int4_group(const float (&x)[16], uint2 &packed, float &s, float &z,
                                           float &da, float &db)
{
    float lo = x[0], hi = x[0];
#pragma unroll
    for (int i = 1; i < 16; ++i) { lo = fminf(lo, x[i]); hi = fmaxf(hi, x[i]); }
    float range = fmaxf(__fsub_rn(hi, lo), 1e-8f);
    s = __fdiv_rn(range, 15.0f);
    z = lo;
    float diff[16];
    unsigned code[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        float r = rintf(__fdiv_rn(__fsub_rn(x[i], z), s));
        r = fminf(fmaxf(r, 0.0f), 15.0f);
        code[i] = (unsigned)r;
        float deq = __fadd_rn(__fmul_rn(r, s), z);
        diff[i] = __fsub_rn(x[i], deq);
    }
    unsigned w0 = 0, w1 = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        w0 |= (code[2 * j] | (code[2 * j + 1] << 4)) << (8 * j);
        w1 |= (code[8 + 2 * j] | (code[8 + 2 * j + 1] << 4)) << (8 * j);
    }
    packed = make_uint2(w0, w1);
    sumsq16(diff, da, db);
}

// Quantise one complete block.  ksrc/vsrc: 16 rows of 128 elements of T.
template <typename T>
__device__ void quantize_one_block(const cqa_cache &c, int kv, long blk, const T *ksrc, const T *vsrc,
                                   bool do_keys, bool do_values, bool eta_mean, bool write_nu,
                                   BlockQuantSmem &sm)
{
    const int tid = threadIdx.x;
    const long row0 = (long)kv * c.cap_tokens + blk * BS;
    const long bidx = (long)kv * c.max_blocks + blk;

    if (do_keys) {
        const int ch = tid;
        float x[BS];
#pragma unroll
        for (int t = 0; t < BS; ++t) x[t] = Cvt<T>::to_f(ksrc[t * D + ch]);
        float lo = x[0], hi = x[0];
#pragma unroll
        for (int t = 1; t < BS; ++t) { lo = fminf(lo, x[t]); hi = fmaxf(hi, x[t]); }
        float range = fmaxf(__fsub_rn(hi, lo), 1e-8f);
        float s = __fdiv_rn(range, 255.0f);
        float z = __fdiv_rn(__fadd_rn(lo, hi), 2.0f);
#pragma unroll
        for (int t = 0; t < BS; ++t) {
            float r = rintf(__fdiv_rn(__fsub_rn(x[t], z), s));
            r = fminf(fmaxf(r, -128.0f), 127.0f);
            c.keys_int8[(row0 + t) * D + ch] = (int8_t)r;
        }
        c.keys_scale[bidx * D + ch] = s;
        c.keys_zero_points[bidx * D + ch] = z;
        sm.scale[ch] = s;
        if (c.sigma_max) atomicMax(reinterpret_cast<int *>(c.sigma_max) + kv * D + ch, __float_as_int(s));
    }
    if (do_values) {
        const int t = tid >> 3, g = tid & 7;
        float xm[16], x[16];
        float a[8], b[8];
        load8<T>(vsrc + t * D + g * GS, a);
        load8<T>(vsrc + t * D + g * GS + 8, b);
#pragma unroll
        for (int i = 0; i < 8; ++i) { xm[i] = a[i]; xm[i + 8] = b[i]; }
        // values.to(float16) before quantising (prefill and deferred block paths)
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = __half2float(__float2half_rn(xm[i]));
        uint2 packed;
        float s, z, da, db, xa, xb, na, nb;
        int4_group(x, packed, s, z, da, db);
        sumsq16(x, xa, xb);
        sumsq16(xm, na, nb);
        const long row = row0 + t;
        *reinterpret_cast<uint2 *>(c.values_int4_packed + row * (D / 2) + g * 8) = packed;
        c.values_int4_scales[row * NG + g] = __half_as_ushort(__float2half_rn(s));
        c.values_int4_zeros[row * NG + g] = __half_as_ushort(__float2half_rn(z));
        float ae = __fsqrt_rn(group8_sum(da, db));
        float xn = fmaxf(__fsqrt_rn(group8_sum(xa, xb)), 1e-6f);
        float vn = __fsqrt_rn(group8_sum(na, nb));
        if (g == 0) {
            sm.tok_err[t] = __fdiv_rn(ae, xn);
            sm.tok_vnorm[t] = vn;
        }
    }
    __syncthreads();
    if (do_keys && tid < 32) {
        const int L = tid & 15;
        float a[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] = sm.scale[8 * L + i];
        float n2 = hw_sum(chain8(a, a));
        if (tid == 0) {
            float delta = __fdiv_rn(__fsqrt_rn(n2), 127.0f);
            c.correction[bidx] = cexp(__fmul_rn(2.0f, delta));
        }
    }
    if (do_values && tid == 0) {
        float p[BS];
        float mx = sm.tok_err[0], vmx = sm.tok_vnorm[0];
#pragma unroll
        for (int i = 0; i < BS; ++i) {
            p[i] = sm.tok_err[i];
            mx = fmaxf(mx, p[i]);
            vmx = fmaxf(vmx, sm.tok_vnorm[i]);
        }
#pragma unroll
        for (int s = 8; s >= 1; s >>= 1)
#pragma unroll
            for (int i = 0; i < s; ++i) p[i] = __fadd_rn(p[i], p[i + s]);
        c.values_int4_errors[bidx] = eta_mean ? __fdiv_rn(p[0], 16.0f) : mx;
        c.values_int4_error_sums[bidx] = p[0];
        c.values_int4_error_counts[bidx] = BS;
        if (write_nu) c.values_norm_max[bidx] = vmx;
    }
    __syncthreads();
}

// ---------------------------------------------------------------- block encoder (prefill)
//
// encode_blocks_kernel: a warp encodes a run of 16-token blocks of one KV head, keys and values alternately.
// A block's rows are contiguous in every array, so they travel by bulk copies: rows into one of two shared-memory
// slots while the other is worked on, from there to Tier 2 unchanged, and the codes, scales and zero points from
// staging areas to HBM (10 copies per block, issued by one lane).  In registers half warp hw holds the tokens 2j + hw,
// lane L the channels 8L..8L+7.  The per-channel maxima of the scales stay in registers over the run and reach the
// global array by an atomic only where they raise it.
//
// The loops over the rows are rolled: unrolled (twice or fully, 168 to 128 registers) the kernel is bound by
// instruction fetch, 250 to 300 us for 65536 bf16 tokens x 8 KV heads against 170 rolled with 16 warps per SM
// (771 us for the form before, a thread per channel with 2-byte accesses, a division per element and 128 atomics per
// block).  HBM bound of that size: 105 us; what is left is instruction issue, about 3700 per block.
//
// rint((x - z) / s) is taken from a product with an approximate reciprocal.  The two can only differ where the
// quotient is near a half-integer (the product is off by at most 4 * 2^-24 of itself), and there the division's
// rounded result is decided from the exact residual (x - z) - h * s (tie_round); bf16 and fp16 rows hit exact
// half-integers at 2 to 4 elements in 1000, and a key channel's smallest element always lands on -127.5, so that one's
// code is found once per channel.
constexpr int ENC_WARPS = 4;
constexpr float ENC_MAGIC = 12582912.0f;      // 1.5 * 2^23: adding it rounds to the nearest integer (ties to even)
constexpr float ENC_TIE_KEYS = 0.5f - 3.1e-5f;    // |q| <= 128: 128 * 4 * 2^-24 = 3.05e-5
constexpr float ENC_TIE_VALUES = 0.5f - 4e-6f;    // |q| <= 15.5: 3.7e-6

template <typename T>
struct EncLayout {
    static constexpr int SLOTS = 2;
    static constexpr int IN = BS * D * (int)sizeof(T);
    static constexpr int K_CODES = SLOTS * IN, K_SCALE = K_CODES + BS * D, K_ZERO = K_SCALE + D * 4;
    static constexpr int V_CODES = K_ZERO + D * 4, V_SCALE = V_CODES + BS * D / 2, V_ZERO = V_SCALE + BS * NG * 2;
    static constexpr int WARP = V_ZERO + BS * NG * 2;
    static constexpr int TOTAL = ENC_WARPS * (WARP + 8 * 4);      // + mbarriers
    static constexpr int CTAS = sizeof(T) == 2 ? 4 : 2;           // resident per SM
};

__device__ __forceinline__ void bulk_store(void *dst_gmem, unsigned src_addr, unsigned bytes)
{
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst_gmem), "r"(src_addr), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ float approx_rcp(float x)
{
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float min_nan(float a, float b)     // NaN if either is
{
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
// rint of the correctly rounded d / s, given q within a few ulps of d / s (|q| < 1024, s finite).  With h the
// half-integer above floor(q), the residual d - h * s is exact where it decides anything (d and h * s agree in all
// but their last bits); the rounded quotient is h itself when the residual is within half a gap of h, and then
// rounds to even, otherwise the residual's sign tells the side.  (The gap below 0.5 is half the gap above.)
__device__ __forceinline__ float tie_round(float d, float s, float q)
{
    const float h = floorf(q) + 0.5f;
    const float rho = __fmaf_rn(-h, s, d);
    float gap = s * (__uint_as_float(__float_as_uint(h) & 0x7F800000u) * 5.9604644775390625e-08f);   // s * ulp(h) / 2
    if (fabsf(h) == 0.5f && (rho < 0.0f) != (h < 0.0f)) gap *= 0.5f;
    return fabsf(rho) <= gap ? rintf(h) : h + copysignf(0.5f, rho);
}

// a - b with one rounding, as a fused multiply-add: the packed add has no negated operands.
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }

// Eight elements of a row: t[i] = ENC_MAGIC + clamp(rint((x - z) / s)); the code is in the low bits of t.  KEYS:
// elements whose difference equals d0 (the channel's smallest) take t0.
template <bool KEYS>
__device__ __forceinline__ void quant_row(const float2 (&x)[4], const float2 (&z)[4], const float2 (&s)[4], const float2 (&inv)[4],
                                          const float2 (&d0)[4], const float2 (&t0)[4], bool exact, float2 (&t)[4])
{
    constexpr float HI = KEYS ? 127.0f : 15.0f, LO = KEYS ? -128.0f : 0.0f, TIE = KEYS ? ENC_TIE_KEYS : ENC_TIE_VALUES;
    const float2 m = make_float2(ENC_MAGIC, ENC_MAGIC), nm = make_float2(-ENC_MAGIC, -ENC_MAGIC);
    float2 d[4], q[4];
    bool fx[4], fy[4];                    // near a half-integer (or NaN)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        d[i] = sub2(x[i], z[i]);
        q[i] = __fmul2_rn(d[i], inv[i]);
        if (KEYS) { q[i].x = min_nan(q[i].x, HI); q[i].y = min_nan(q[i].y, HI); }     // 127.5 may round to 128
        t[i] = __fadd2_rn(q[i], m);
        const float2 e = sub2(q[i], __fadd2_rn(t[i], nm));
        fx[i] = !(fabsf(e.x) <= TIE);
        fy[i] = !(fabsf(e.y) <= TIE);
        if (KEYS) {
            const bool lx = d[i].x == d0[i].x, ly = d[i].y == d0[i].y;
            fx[i] = fx[i] && !lx;
            fy[i] = fy[i] && !ly;
            t[i].x = lx ? t0[i].x : t[i].x;
            t[i].y = ly ? t0[i].y : t[i].y;
        }
    }
    bool bad = exact;
    if (__any_sync(FULL, fx[0] || fy[0] || fx[1] || fy[1] || fx[2] || fy[2] || fx[3] || fy[3])) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (__any_sync(FULL, fx[i] || fy[i])) {
                const float rx = tie_round(d[i].x, s[i].x, q[i].x), ry = tie_round(d[i].y, s[i].y, q[i].y);
                t[i].x = fx[i] ? fminf(fmaxf(rx, LO), HI) + ENC_MAGIC : t[i].x;
                t[i].y = fy[i] ? fminf(fmaxf(ry, LO), HI) + ENC_MAGIC : t[i].y;
                bad |= (fx[i] && !(fabsf(q[i].x) < 1024.0f)) || (fy[i] && !(fabsf(q[i].y) < 1024.0f));
            }
        }
    }
    if (__any_sync(FULL, bad)) {    // NaN or infinite elements, or a scale whose reciprocal is not normal
        if (bad) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                t[i].x = fminf(fmaxf(rintf(__fdiv_rn(__fsub_rn(x[i].x, z[i].x), s[i].x)), LO), HI) + ENC_MAGIC;
                t[i].y = fminf(fmaxf(rintf(__fdiv_rn(__fsub_rn(x[i].y, z[i].y), s[i].y)), LO), HI) + ENC_MAGIC;
            }
        }
    }
}
__device__ __forceinline__ void to_pairs(const float (&x)[8], float2 (&p)[4])
{
#pragma unroll
    for (int i = 0; i < 4; ++i) p[i] = make_float2(x[2 * i], x[2 * i + 1]);
}
// chain8 on packed operands (even channels in .x, odd ones in .y).
__device__ __forceinline__ float chain8_pairs(const float2 (&a)[4])
{
    float2 p = __ffma2_rn(a[0], a[0], make_float2(0.0f, 0.0f));
    p = __ffma2_rn(a[1], a[1], p);
    p = __ffma2_rn(a[2], a[2], p);
    p = __ffma2_rn(a[3], a[3], p);
    return __fadd_rn(p.x, p.y);
}
// Element-wise extremes of raw rows; two-byte types stay packed.
__device__ __forceinline__ void raw_minmax(const Raw8<float> &x, Raw8<float> &lo, Raw8<float> &hi)
{
    const float *a = &x.a.x, *b = &x.b.x;
    float *la = &lo.a.x, *lb = &lo.b.x, *ha = &hi.a.x, *hb = &hi.b.x;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        la[i] = fminf(la[i], a[i]); ha[i] = fmaxf(ha[i], a[i]);
        lb[i] = fminf(lb[i], b[i]); hb[i] = fmaxf(hb[i], b[i]);
    }
}
template <typename T2V>
__device__ __forceinline__ void words_minmax(const uint4 &x, uint4 &lo, uint4 &hi)
{
    const T2V *a = reinterpret_cast<const T2V *>(&x);
    T2V *l = reinterpret_cast<T2V *>(&lo), *h = reinterpret_cast<T2V *>(&hi);
#pragma unroll
    for (int i = 0; i < 4; ++i) { l[i] = __hmin2(l[i], a[i]); h[i] = __hmax2(h[i], a[i]); }
}
__device__ __forceinline__ void raw_minmax(const Raw8<__half> &x, Raw8<__half> &lo, Raw8<__half> &hi) { words_minmax<__half2>(x.v, lo.v, hi.v); }
__device__ __forceinline__ void raw_minmax(const Raw8<__nv_bfloat16> &x, Raw8<__nv_bfloat16> &lo, Raw8<__nv_bfloat16> &hi) { words_minmax<__nv_bfloat162>(x.v, lo.v, hi.v); }
template <typename T>
__device__ __forceinline__ Raw8<T> raw_shfl_xor(const Raw8<T> &r, int o)
{
    Raw8<T> out;
    const unsigned *a = reinterpret_cast<const unsigned *>(&r);
    unsigned *b = reinterpret_cast<unsigned *>(&out);
#pragma unroll
    for (int i = 0; i < (int)(sizeof(Raw8<T>) / 4); ++i) b[i] = __shfl_xor_sync(FULL, a[i], o);
    return out;
}

// Keys of one block: `rows` in shared memory -> codes, scales, zero points in the staging area, correction in HBM.
template <typename T>
__device__ __forceinline__ void encode_keys(const cqa_cache &c, long bidx, const T *rows, char *stage, float (&smax)[8], int hw, int L)
{
    using LY = EncLayout<T>;
    const T *mine = rows + hw * D + 8 * L;
    Raw8<T> lo = raw_load8<T>(mine), hi = lo;
#pragma unroll
    for (int j = 1; j < 8; ++j) raw_minmax(raw_load8<T>(mine + 2 * j * D), lo, hi);
    raw_minmax(raw_shfl_xor(lo, 16), lo, hi);
    raw_minmax(raw_shfl_xor(hi, 16), lo, hi);
    float lf[8], hf[8];
    raw_to_f(lo, lf);
    raw_to_f(hi, hf);
    float2 s[4], z[4], inv[4], d0[4], t0[4];
    bool exact = false;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        float *sp = &s[i >> 1].x + (i & 1), *zp = &z[i >> 1].x + (i & 1);
        *sp = __fdiv_rn(fmaxf(__fsub_rn(hf[i], lf[i]), 1e-8f), 255.0f);
        *zp = __fmul_rn(__fadd_rn(lf[i], hf[i]), 0.5f);
        const float iv = approx_rcp(*sp), d = __fsub_rn(lf[i], *zp);
        *(&inv[i >> 1].x + (i & 1)) = iv;
        *(&d0[i >> 1].x + (i & 1)) = d;
        *(&t0[i >> 1].x + (i & 1)) = fminf(fmaxf(tie_round(d, *sp, d * iv), -128.0f), 127.0f) + ENC_MAGIC;
        exact |= !(*sp < 1e30f);
        smax[i] = fmaxf(smax[i], *sp);
    }
    {
        float4 *dst = reinterpret_cast<float4 *>(stage + (hw ? LY::K_ZERO : LY::K_SCALE)) + 2 * L;
#pragma unroll
        for (int i = 0; i < 2; ++i)
            dst[i] = make_float4(hw ? z[2 * i].x : s[2 * i].x, hw ? z[2 * i].y : s[2 * i].y, hw ? z[2 * i + 1].x : s[2 * i + 1].x,
                                 hw ? z[2 * i + 1].y : s[2 * i + 1].y);
    }
    char *codes = stage + LY::K_CODES + hw * D + 8 * L;
#pragma unroll 1
    for (int j = 0; j < 8; ++j) {
        float x[8];
        float2 x2[4], t[4];
        raw_to_f(raw_load8<T>(mine + 2 * j * D), x);
        to_pairs(x, x2);
        quant_row<true>(x2, z, s, inv, d0, t0, exact, t);
        const unsigned w0 = __byte_perm(__byte_perm(__float_as_uint(t[0].x), __float_as_uint(t[0].y), 0x0040),
                                        __byte_perm(__float_as_uint(t[1].x), __float_as_uint(t[1].y), 0x0040), 0x5410);
        const unsigned w1 = __byte_perm(__byte_perm(__float_as_uint(t[2].x), __float_as_uint(t[2].y), 0x0040),
                                        __byte_perm(__float_as_uint(t[3].x), __float_as_uint(t[3].y), 0x0040), 0x5410);
        *reinterpret_cast<uint2 *>(codes + 2 * j * D) = make_uint2(w0, w1);
    }
    const float n2 = hw_sum(chain8_pairs(s));
    if (hw == 0 && L == 0) c.correction[bidx] = cexp(__fmul_rn(2.0f, __fdiv_rn(__fsqrt_rn(n2), 127.0f)));
}

// Values of one block: INT4 codes, scales and zeros into the staging area (when the cache holds INT4 values), error
// annotations and nu_b in HBM.
template <typename T>
__device__ __forceinline__ void encode_values(const cqa_cache &c, long bidx, const T *rows, char *stage, int hw, int L)
{
    using LY = EncLayout<T>;
    constexpr bool is_half = std::is_same<T, __half>::value;
    const bool int4 = c.values_int4_packed != nullptr;
    const T *mine = rows + hw * D + 8 * L;
    // 16-lane sums in the fixed order (strides 8, 4, 2, 1) of eight tokens at once: a lane keeps the tokens with the
    // bits of its own number, so it ends with token 2 * (L >> 1) + hw.  The stride-8 step is applied to tokens j and
    // j + 4 as soon as both are there.
    float da[4] = {}, xa[4] = {}, na[4] = {};
    const bool up = (L & 8) != 0;
#pragma unroll 1
    for (int jj = 0; jj < 4; ++jj) {
        float cn[2] = {}, cd[2] = {}, cx[2] = {};
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
            const int j = jj + 4 * half;
            float xm[8];
            float2 x2[4];
            raw_to_f(raw_load8<T>(mine + 2 * j * D), xm);
            to_pairs(xm, x2);
            const float n_ = chain8_pairs(x2);
            float d_ = 0.0f, x_ = n_;
            if (int4) {
                __half2 hx[4];          // the INT4 codes quantise values.to(float16)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    hx[i] = __float22half2_rn(x2[i]);
                    if (!is_half) x2[i] = __half22float2(hx[i]);
                }
                __half2 l2 = __hmin2(__hmin2(hx[0], hx[1]), __hmin2(hx[2], hx[3]));
                __half2 h2 = __hmax2(__hmax2(hx[0], hx[1]), __hmax2(hx[2], hx[3]));
                l2 = __hmin2(l2, __lowhigh2highlow(l2));
                h2 = __hmax2(h2, __lowhigh2highlow(h2));
                // the other eight channels of the group
                const __half2 mine2 = __lows2half2(l2, h2);
                const __half2 other = __shfl_xor_sync(FULL, mine2, 1);
                const float lo = __low2float(__hmin2(mine2, other)), hi = __high2float(__hmax2(mine2, other));
                const float s = __fdiv_rn(fmaxf(__fsub_rn(hi, lo), 1e-8f), 15.0f);
                const float iv = approx_rcp(s);
                float2 z4[4], s4[4], iv4[4], t[4], r[4], diff[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) { z4[i] = make_float2(lo, lo); s4[i] = make_float2(s, s); iv4[i] = make_float2(iv, iv); }
                quant_row<false>(x2, z4, s4, iv4, z4, z4, !(s < 1e30f), t);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    r[i] = __fadd2_rn(t[i], make_float2(-ENC_MAGIC, -ENC_MAGIC));
                    // scalar products: a packed product and the packed add behind it are merged into one rounding
                    const float2 deq = __fadd2_rn(make_float2(__fmul_rn(r[i].x, s), __fmul_rn(r[i].y, s)), z4[i]);
                    diff[i] = sub2(x2[i], deq);
                }
                d_ = chain8_pairs(diff);
                if (!is_half) x_ = chain8_pairs(x2);
                // eight codes as two 16-bit numbers, exact in float
                const float a = fmaf(fmaf(r[1].y, 16.0f, r[1].x), 256.0f, fmaf(r[0].y, 16.0f, r[0].x));
                const float b = fmaf(fmaf(r[3].y, 16.0f, r[3].x), 256.0f, fmaf(r[2].y, 16.0f, r[2].x));
                const int row = 2 * j + hw;
                *reinterpret_cast<unsigned *>(stage + LY::V_CODES + row * (D / 2) + 4 * L) =
                    __byte_perm(__float_as_uint(a + 8388608.0f), __float_as_uint(b + 8388608.0f), 0x5410);
                // even lanes store the group's scale, odd lanes its zero
                reinterpret_cast<__half *>(stage + ((L & 1) ? LY::V_ZERO : LY::V_SCALE))[row * NG + (L >> 1)] =
                    __float2half_rn((L & 1) ? lo : s);
            }
            if (half == 0) { cn[0] = n_; cd[0] = d_; cx[0] = x_; } else { cn[1] = n_; cd[1] = d_; cx[1] = x_; }
        }
        const auto fold = [&](const float (&v)[2]) {
            return __fadd_rn(up ? v[1] : v[0], __shfl_xor_sync(FULL, up ? v[0] : v[1], 8));
        };
        const float fn = fold(cn), fd = fold(cd), fx = is_half ? fn : fold(cx);
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (i == jj) { na[i] = fn; da[i] = fd; xa[i] = fx; }
    }
    const auto finish = [&](float (&a)[4]) {
#pragma unroll
        for (int w = 2; w >= 1; w >>= 1) {
            const bool u = (L & (2 * w)) != 0;
#pragma unroll
            for (int j = 0; j < w; ++j)
                a[j] = __fadd_rn(u ? a[j + w] : a[j], __shfl_xor_sync(FULL, u ? a[j] : a[j + w], 2 * w));
        }
        return __fadd_rn(a[0], __shfl_xor_sync(FULL, a[0], 1));
    };
    // maximum and (token strides 8, 4, 2, 1) sum over the block's tokens
    const float vn = __fsqrt_rn(finish(na));
    float vmx = vn, err = 0.0f, sum = 0.0f;
    if (int4) {
        const float ae = __fsqrt_rn(finish(da));
        const float xn = fmaxf(is_half ? vn : __fsqrt_rn(finish(xa)), 1e-6f);
        err = __fdiv_rn(ae, xn);
        sum = err;
    }
#pragma unroll
    for (int o = 8; o >= 1; o >>= 1) {
        const int x = o == 1 ? 16 : o;     // lane bits 3, 2, 1 number j = token / 2; the half warp is the token's low bit
        vmx = fmaxf(vmx, __shfl_xor_sync(FULL, vmx, x));
        err = fmaxf(err, __shfl_xor_sync(FULL, err, x));
        sum = __fadd_rn(sum, __shfl_xor_sync(FULL, sum, x));
    }
    if (hw == 0 && L == 0) {
        c.values_norm_max[bidx] = vmx;
        if (int4) {
            c.values_int4_errors[bidx] = err;
            c.values_int4_error_sums[bidx] = sum;
            c.values_int4_error_counts[bidx] = BS;
        }
    }
}

// Where token `tok` of KV head kv is copied to: the Tier-2 array itself, or with a slot table (bounded hot tier, whose
// scratch starts empty) the backing array; nullptr when there is neither.
template <typename T>
__device__ __forceinline__ T *t2_copy_rows(void *hot, long hot_rows, const int32_t *slots, void *backing, long backing_rows,
                                           int kv, long tok)
{
    T *base = reinterpret_cast<T *>(slots ? backing : hot);
    return base ? base + ((long)kv * (slots ? backing_rows : hot_rows) + tok) * D : nullptr;
}

// Grid (runs of ENC_WARPS * bpw blocks, KV).  The launches of one prefill touch different memory, so they may overlap
// (programmatic launch); each waits for its predecessor at its end, so that the last one ends after all of them.
template <typename T>
__global__ void __launch_bounds__(ENC_WARPS * 32, EncLayout<T>::CTAS)
encode_blocks_kernel(const __grid_constant__ cqa_cache c, const T *k_src, const T *v_src, long src_rows, long first_block,
                     long n_blocks, int bpw, int copy_t2)
{
    using LY = EncLayout<T>;
    extern __shared__ __align__(128) char esm[];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int kv = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, L = lane & 15, hw = lane >> 4;
    const long b0 = ((long)blockIdx.x * ENC_WARPS + warp) * bpw;
    const int nb = (int)max(0L, min(n_blocks, b0 + bpw) - b0);
    if (nb > 0) {
        char *wsm = esm + warp * LY::WARP;
        uint64_t *bars = reinterpret_cast<uint64_t *>(esm + ENC_WARPS * LY::WARP) + 4 * warp;
        const unsigned wsm_a = smem_u32(wsm), bar_a = smem_u32(bars);
        if (lane == 0) {
            for (int i = 0; i < LY::SLOTS; ++i) mbar_init(bars + i, 1);
            mbar_init_fence();
        }
        __syncwarp();
        const T *ks = k_src + ((long)kv * src_rows + b0 * BS) * D;
        const T *vs = v_src + ((long)kv * src_rows + b0 * BS) * D;
        T *kd = copy_t2 ? t2_copy_rows<T>(c.keys_t2, c.keys_t2_rows, c.key_slots, c.keys_t2_backing, c.t2_backing_rows, kv, (first_block + b0) * BS) : nullptr;
        T *vd = copy_t2 ? t2_copy_rows<T>(c.values_t2, c.values_t2_rows, c.value_slots, c.values_t2_backing, c.t2_backing_rows, kv, (first_block + b0) * BS) : nullptr;
        const bool bulk_in = (((uintptr_t)ks | (uintptr_t)vs) & 15) == 0;
        const long blk0 = first_block + b0;
        const bool int4 = c.values_int4_packed != nullptr;
        float smax[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) smax[i] = 0.0f;
        // unit u: keys (even u) or values (odd u) of block b0 + u / 2, in slot u mod SLOTS
        const auto fetch = [&](int u) {
            if (lane == 0 && u < 2 * nb) {
                const int slot = u % LY::SLOTS;
                mbar_arrive_expect_tx(bar_a + 8 * slot, LY::IN);
                bulk_copy_g2s(wsm_a + slot * LY::IN, ((u & 1) ? vs : ks) + (long)(u >> 1) * BS * D, LY::IN, bar_a + 8 * slot);
            }
        };
        if (bulk_in)
            for (int u = 0; u < LY::SLOTS - 1; ++u) fetch(u);
        int slot = 0, phase = 0;
#pragma unroll 1
        for (int u = 0; u < 2 * nb; ++u) {
            const T *rows = reinterpret_cast<const T *>(wsm + slot * LY::IN);
            const long blk = blk0 + (u >> 1), bidx = (long)kv * c.max_blocks + blk, row0 = (long)kv * c.cap_tokens + blk * BS;
            // every store but the last group's has left shared memory: the previous unit's slot and the staging area
            // of the unit before that are free
            if (lane == 0) bulk_wait_read<1>();
            __syncwarp();
            if (bulk_in) {
                fetch(u + LY::SLOTS - 1);
                mbar_wait(bar_a + 8 * slot, (unsigned)phase);
            } else {
                const T *src = ((u & 1) ? vs : ks) + (long)(u >> 1) * BS * D;
                for (int i = lane; i < BS * D; i += 32) const_cast<T *>(rows)[i] = src[i];
                fence_async_smem();
                __syncwarp();
            }
            if (lane == 0) {
                T *dst = (u & 1) ? vd : kd;
                if (dst) bulk_store(dst + (long)(u >> 1) * BS * D, wsm_a + slot * LY::IN, LY::IN);
                bulk_commit();
            }
            if (u & 1) encode_values<T>(c, bidx, rows, wsm, hw, L);
            else encode_keys<T>(c, bidx, rows, wsm, smax, hw, L);
            fence_async_smem();
            __syncwarp();
            if (lane == 0) {
                if (!(u & 1)) {
                    bulk_store(c.keys_int8 + row0 * D, wsm_a + LY::K_CODES, BS * D);
                    bulk_store(c.keys_scale + bidx * D, wsm_a + LY::K_SCALE, D * 4);
                    bulk_store(c.keys_zero_points + bidx * D, wsm_a + LY::K_ZERO, D * 4);
                } else if (int4) {
                    bulk_store(c.values_int4_packed + row0 * (D / 2), wsm_a + LY::V_CODES, BS * D / 2);
                    bulk_store(c.values_int4_scales + row0 * NG, wsm_a + LY::V_SCALE, BS * NG * 2);
                    bulk_store(c.values_int4_zeros + row0 * NG, wsm_a + LY::V_ZERO, BS * NG * 2);
                }
                bulk_commit();
            }
            if (++slot == LY::SLOTS) { slot = 0; phase ^= 1; }
        }
        if (c.sigma_max && hw == 0) {
            float *sm = c.sigma_max + kv * D + 8 * L;
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (smax[i] > __ldcg(sm + i)) atomicMax(reinterpret_cast<int *>(sm + i), __float_as_int(smax[i]));
        }
        if (lane == 0) bulk_wait_all();
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// The ragged tail of a prefill: n_tail < 16 tokens from first_pos (a block boundary), with the effect of appending
// them one by one (append_token_body), by CTA x = 0 of each KV head; a token per half warp.  CTAs x >= 1 write the
// state of an empty cache into the reserve behind the tail's block when `init` is set (the caller's arrays are then
// uninitialised memory): one launch instead of a fill per array.
constexpr int TAIL_INIT_CTAS = 8;
template <typename T>
__device__ __forceinline__ float round_t2(float x, int t2_dtype)
{
    if (t2_dtype == CQA_F16) return __half2float(__float2half_rn(x));
    if (t2_dtype == CQA_BF16) return __bfloat162float(__float2bfloat16_rn(x));
    return x;
}
__device__ __forceinline__ void fill16(void *base, long from, long to, int part, int parts)   // bytes [from, to), 16-byte units
{
    char *p = reinterpret_cast<char *>(base);
    if (p == nullptr) return;
    for (long i = from + 16L * (part * (long)blockDim.x + threadIdx.x); i < to; i += 16L * parts * blockDim.x)
        *reinterpret_cast<uint4 *>(p + i) = make_uint4(0u, 0u, 0u, 0u);
}
__device__ __forceinline__ void fill_words(void *base, long from, long to, unsigned v, int part, int parts)
{
    unsigned *p = reinterpret_cast<unsigned *>(base);
    if (p == nullptr) return;
    for (long i = from + part * (long)blockDim.x + threadIdx.x; i < to; i += (long)parts * blockDim.x) p[i] = v;
}
// Rows [tok, tok_end) and blocks [blk, blk_end) of KV head kv as an empty cache holds them.
__device__ __forceinline__ void clear_reserve(const cqa_cache &c, int kv, long tok, long tok_end, long blk, long blk_end,
                                              int part, int parts)
{
    const long r = (long)kv * c.cap_tokens, g = (long)kv * c.max_blocks, esz = c.t2_dtype == CQA_F32 ? 4 : 2;
    fill16(c.keys_int8, (r + tok) * D, (r + tok_end) * D, part, parts);
    fill16(c.values_int4_packed, (r + tok) * (D / 2), (r + tok_end) * (D / 2), part, parts);
    fill16(c.values_int4_scales, (r + tok) * NG * 2, (r + tok_end) * NG * 2, part, parts);
    fill16(c.values_int4_zeros, (r + tok) * NG * 2, (r + tok_end) * NG * 2, part, parts);
    fill16(c.keys_scale, (g + blk) * D * 4, (g + blk_end) * D * 4, part, parts);
    fill16(c.keys_zero_points, (g + blk) * D * 4, (g + blk_end) * D * 4, part, parts);
    fill_words(c.correction, g + blk, g + blk_end, __float_as_uint(1.0f), part, parts);
    fill_words(c.values_int4_errors, g + blk, g + blk_end, 0u, part, parts);
    fill_words(c.values_int4_error_sums, g + blk, g + blk_end, 0u, part, parts);
    fill_words(c.values_int4_error_counts, g + blk, g + blk_end, 0u, part, parts);
    fill_words(c.values_norm_max, g + blk, g + blk_end, 0u, part, parts);
    const long rk = (long)kv * c.keys_t2_rows, rv = (long)kv * c.values_t2_rows;
    if (!c.key_slots) fill16(c.keys_t2, (rk + tok) * D * esz, (rk + min(tok_end, (long)c.keys_t2_rows)) * D * esz, part, parts);
    if (!c.value_slots) fill16(c.values_t2, (rv + tok) * D * esz, (rv + min(tok_end, (long)c.values_t2_rows)) * D * esz, part, parts);
}
template <typename T>
__global__ void __launch_bounds__(256) prefill_tail_kernel(const __grid_constant__ cqa_cache c, const T *k_src, const T *v_src,
                                                          long src_rows, long first_pos, int n_tail, int defer_int4, int init)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int kv = blockIdx.y, tid = threadIdx.x;
    const long blk = first_pos / BS;
    const long clear_tok = first_pos + (n_tail ? BS : 0), clear_blk = blk + (n_tail ? 1 : 0);
    __shared__ float s_err[BS], s_vn[BS];
    if (blockIdx.x > 0) {
        clear_reserve(c, kv, clear_tok, c.cap_tokens, clear_blk, c.max_blocks, (int)blockIdx.x - 1, (int)gridDim.x - 1);
    } else if (n_tail > 0) {
        if (init) {
            clear_reserve(c, kv, first_pos, min(first_pos + BS, (long)c.cap_tokens), blk, blk + 1, 0, 1);
            __syncthreads();
        }
        const int t = tid >> 4, L = tid & 15;
        const bool live = t < n_tail;
        const long pos = first_pos + t, bidx = (long)kv * c.max_blocks + blk;
        float kx[8], vx[8];
        if (live) {
            const long o = ((long)kv * src_rows + pos) * D + 8 * L;
#pragma unroll
            for (int i = 0; i < 8; ++i) {     // element loads: the source may start anywhere
                kx[i] = round_t2<T>(Cvt<T>::to_f(k_src[o + i]), c.t2_dtype);
                vx[i] = round_t2<T>(Cvt<T>::to_f(v_src[o + i]), c.t2_dtype);
            }
            // Tier-2 rows: the mirror, or the backing array and the slot when the block is resident
            long krow = pos, vrow = pos;
            if (c.key_slots) { const int s = c.key_slots[blk]; krow = s < 0 ? -1 : (long)s * BS + t; }
            if (c.value_slots) { const int s = c.value_slots[blk]; vrow = s < 0 ? -1 : (long)s * BS + t; }
            const auto put = [&](void *base, long rows, long row, const float (&x)[8]) {
                if (base == nullptr || row < 0) return;
                const long at = ((long)kv * rows + row) * D + 8 * L;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (c.t2_dtype == CQA_F32) reinterpret_cast<float *>(base)[at + i] = x[i];
                    else if (c.t2_dtype == CQA_F16) reinterpret_cast<__half *>(base)[at + i] = __float2half_rn(x[i]);
                    else reinterpret_cast<__nv_bfloat16 *>(base)[at + i] = __float2bfloat16_rn(x[i]);
                }
            };
            put(c.keys_t2, c.keys_t2_rows, krow, kx);
            put(c.values_t2, c.values_t2_rows, vrow, vx);
            if (c.key_slots) put(c.keys_t2_backing, c.t2_backing_rows, pos, kx);
            if (c.value_slots) put(c.values_t2_backing, c.t2_backing_rows, pos, vx);
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) vx[i] = 0.0f;
        }
        const bool int4 = c.values_int4_packed != nullptr && !defer_int4;
        float2 x2[4];
        to_pairs(vx, x2);
        const float vn = __fsqrt_rn(hw_sum(chain8_pairs(x2)));
        float err = 0.0f;
        if (int4) {
            float lo = x2[0].x, hi = x2[0].x;
#pragma unroll
            for (int i = 0; i < 4; ++i) { lo = fminf(lo, fminf(x2[i].x, x2[i].y)); hi = fmaxf(hi, fmaxf(x2[i].x, x2[i].y)); }
            lo = fminf(lo, __shfl_xor_sync(FULL, lo, 1));
            hi = fmaxf(hi, __shfl_xor_sync(FULL, hi, 1));
            const float s = __fdiv_rn(fmaxf(__fsub_rn(hi, lo), 1e-8f), 15.0f);
            float diff[8];
            unsigned w = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float r = fminf(fmaxf(rintf(__fdiv_rn(__fsub_rn(vx[i], lo), s)), 0.0f), 15.0f);
                w |= (unsigned)r << (4 * i);
                diff[i] = __fsub_rn(vx[i], __fadd_rn(__fmul_rn(r, s), lo));
            }
            float2 d2[4];
            to_pairs(diff, d2);
            const float ae = __fsqrt_rn(hw_sum(chain8_pairs(d2)));
            err = __fdiv_rn(ae, fmaxf(vn, 1e-6f));
            if (live) {
                const long row = (long)kv * c.cap_tokens + pos;
                *reinterpret_cast<unsigned *>(c.values_int4_packed + row * (D / 2) + 4 * L) = w;
                uint16_t *dst = (L & 1) ? c.values_int4_zeros : c.values_int4_scales;
                dst[row * NG + (L >> 1)] = __half_as_ushort(__float2half_rn((L & 1) ? lo : s));
            }
        }
        if (L == 0) { s_err[t] = err; s_vn[t] = vn; }
        // the INT8 rows behind the first of an open block are poisoned
        if (t >= 1 && pos < c.cap_tokens)
            *reinterpret_cast<uint2 *>(c.keys_int8 + ((long)kv * c.cap_tokens + pos) * D + 8 * L) = make_uint2(0x81818181u, 0x81818181u);
        __syncthreads();
        if (tid == 0) {
            float nu = 0.0f, sum = 0.0f, mx = 0.0f;
            for (int i = 0; i < n_tail; ++i) {
                nu = fmaxf(nu, s_vn[i]);
                sum = __fadd_rn(sum, s_err[i]);     // running sum in token order
                mx = fmaxf(mx, s_err[i]);
            }
            c.values_norm_max[bidx] = nu;
            if (int4) {
                c.values_int4_errors[bidx] = mx;
                c.values_int4_error_sums[bidx] = sum;
                c.values_int4_error_counts[bidx] = n_tail;
            }
        }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Fused append-and-quantise of one token.  Grid: KV CTAs of 128 threads.
template <typename T2>
__device__ __forceinline__ void append_token_body(const cqa_cache &c, const void *k_new, const void *v_new, int src_dtype,
                                                  long pos, int defer_int4)
{
    __shared__ BlockQuantSmem sm;
    __shared__ float s_v[D];
    const int kv = blockIdx.x, tid = threadIdx.x;
    const long blk = pos / BS;
    const int pib = (int)(pos % BS);
    const long bidx = (long)kv * c.max_blocks + blk;
    grid_dependency_wait();

    long krow = pos, vrow = pos;
    if (c.key_slots) { int s = c.key_slots[blk]; krow = s < 0 ? -1 : (long)s * BS + pib; }
    if (c.value_slots) { int s = c.value_slots[blk]; vrow = s < 0 ? -1 : (long)s * BS + pib; }

    T2 kq = Cvt<T2>::from_f(load_q(k_new, src_dtype, (long)kv * D + tid));
    T2 vq = Cvt<T2>::from_f(load_q(v_new, src_dtype, (long)kv * D + tid));
    T2 *kt2 = reinterpret_cast<T2 *>(c.keys_t2);
    T2 *vt2 = reinterpret_cast<T2 *>(c.values_t2);
    if (kt2 && krow >= 0) kt2[((long)kv * c.keys_t2_rows + krow) * D + tid] = kq;
    if (vt2 && vrow >= 0) vt2[((long)kv * c.values_t2_rows + vrow) * D + tid] = vq;
    // bounded hot tier: the backing arrays always receive the row (the hot copy above only if the block is resident)
    if (c.key_slots && c.keys_t2_backing)
        reinterpret_cast<T2 *>(c.keys_t2_backing)[((long)kv * c.t2_backing_rows + pos) * D + tid] = kq;
    if (c.value_slots && c.values_t2_backing)
        reinterpret_cast<T2 *>(c.values_t2_backing)[((long)kv * c.t2_backing_rows + pos) * D + tid] = vq;
    s_v[tid] = Cvt<T2>::to_f(vq);
    __syncthreads();

    // nu_b running max with the new token's value norm
    if (tid < 32) {
        const int L = tid & 15;
        float a[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] = s_v[8 * L + i];
        float vn = __fsqrt_rn(hw_sum(chain8(a, a)));
        if (tid == 0) {
            float old = pib == 0 ? 0.0f : c.values_norm_max[bidx];
            c.values_norm_max[bidx] = fmaxf(old, vn);
        }
    }
    // per-token INT4 (only when quantisation is not deferred to block completion)
    if (c.values_int4_packed && !defer_int4 && tid < 32) {
        const int g = tid & 7;
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = s_v[g * GS + i];
        uint2 packed;
        float s, z, da, db, xa, xb;
        int4_group(x, packed, s, z, da, db);
        sumsq16(x, xa, xb);
        float ae = __fsqrt_rn(group8_sum(da, db));
        float xn = fmaxf(__fsqrt_rn(group8_sum(xa, xb)), 1e-6f);
        if (tid < 8) {
            const long row = (long)kv * c.cap_tokens + pos;
            *reinterpret_cast<uint2 *>(c.values_int4_packed + row * (D / 2) + g * 8) = packed;
            c.values_int4_scales[row * NG + g] = __half_as_ushort(__float2half_rn(s));
            c.values_int4_zeros[row * NG + g] = __half_as_ushort(__float2half_rn(z));
            if (tid == 0) {
                float err = __fdiv_rn(ae, xn);
                float osum = pib == 0 ? 0.0f : c.values_int4_error_sums[bidx];
                int ocnt = pib == 0 ? 0 : c.values_int4_error_counts[bidx];
                float oerr = pib == 0 ? 0.0f : c.values_int4_errors[bidx];
                c.values_int4_error_sums[bidx] = __fadd_rn(osum, err);
                c.values_int4_error_counts[bidx] = ocnt + 1;
                c.values_int4_errors[bidx] = fmaxf(oerr, err);
            }
        }
    }
    if (pib == BS - 1) {
        // The block just filled: quantise it from the Tier-2 rows (this CTA wrote the last one).
        __threadfence_block();
        __syncthreads();
        __threadfence();   // the rows may have gone to the backing arrays only
        const T2 *ks = t2_key_block<T2>(c, kv, blk);
        const T2 *vs = t2_value_block<T2>(c, kv, blk);
        if (ks && vs) {
            quantize_one_block<T2>(c, kv, blk, ks, vs, true,
                                   c.values_int4_packed != nullptr && defer_int4 != 0, true, false, sm);
        }
    } else if (pib == 0) {
        // New block opened: poison the not-yet-written INT8 rows.
        const long row0 = (long)kv * c.cap_tokens + pos;
        for (int t = 1; t < BS; ++t)
            if (pos + t < c.cap_tokens) c.keys_int8[(row0 + t) * D + tid] = (int8_t)-127;
    }
}

template <typename T2>
__global__ void __launch_bounds__(128) append_token_kernel(cqa_cache c, const void *k_new, const void *v_new,
                                                          int src_dtype, long pos, int defer_int4)
{
    append_token_body<T2>(c, k_new, v_new, src_dtype, pos, defer_int4);
}

// One token for every sequence of a batch: grid (KV, sequences).
template <typename T2>
__global__ void __launch_bounds__(128) append_token_batched_kernel(const cqa_batch_item *items, int src_dtype)
{
    const cqa_batch_item &it = *stage_batch_item(items + blockIdx.y);
    append_token_body<T2>(it.cache, it.k_new, it.v_new, src_dtype, it.pos, it.defer_int4);
}

// The same with the records as kernel parameters: the CTAs of KV head 0 write them to `dev`, where the other kernels
// of the step read them.  A copy of the records between two steps cost a transfer through the copy engine in the
// middle of a chain of kernels, about 10 us of a batch step.  Parameters grow the launch itself, hence two sizes; beyond 40
// sequences the step is long enough for the copy.
template <int N>
struct BatchRecords {
    cqa_batch_item it[N];
};
constexpr int RECORDS_SMALL = 8, RECORDS_LARGE = 40;
static_assert(sizeof(BatchRecords<RECORDS_LARGE>) + 16 <= 32764, "limit of a kernel's parameters");
template <typename T2, int N>
__global__ void __launch_bounds__(128) append_token_records_kernel(const __grid_constant__ BatchRecords<N> rec, cqa_batch_item *dev, int src_dtype)
{
    grid_dependency_wait();          // the previous step's kernels have read their records
    const cqa_batch_item &it = rec.it[blockIdx.y];
    if (blockIdx.x == 0) {
        const int *from = reinterpret_cast<const int *>(&it);
        int *to = reinterpret_cast<int *>(dev + blockIdx.y);
        for (int i = threadIdx.x; i < (int)(sizeof(cqa_batch_item) / 4); i += blockDim.x) to[i] = from[i];
    }
    append_token_body<T2>(it.cache, it.k_new, it.v_new, src_dtype, it.pos, it.defer_int4);
}

template <typename T2, int N>
static int append_records_n(const cqa_batch_item *items, cqa_batch_item *dev, int n_items, int kv_heads, int src_dtype, cudaStream_t st)
{
    BatchRecords<N> rec;
    memcpy(rec.it, items, (size_t)n_items * sizeof(cqa_batch_item));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)kv_heads, (unsigned)n_items);
    cfg.blockDim = dim3(128);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void *args[] = {&rec, &dev, &src_dtype};
    note_launch();
    return check_cuda(cudaLaunchKernelExC(&cfg, reinterpret_cast<const void *>(append_token_records_kernel<T2, N>), args), "append_token_records_kernel");
}
template <typename T2>
static int append_batched_t(const cqa_batch_item *items, cqa_batch_item *dev, int n_items, int kv_heads, int src_dtype, cudaStream_t st)
{
    if (n_items <= RECORDS_SMALL) return append_records_n<T2, RECORDS_SMALL>(items, dev, n_items, kv_heads, src_dtype, st);
    if (n_items <= RECORDS_LARGE) return append_records_n<T2, RECORDS_LARGE>(items, dev, n_items, kv_heads, src_dtype, st);
    int rc = check_cuda(cudaMemcpyAsync(dev, items, (size_t)n_items * sizeof(cqa_batch_item), cudaMemcpyHostToDevice, st),
                        "copy of the batch records");
    if (rc) return rc;
    return check_cuda(launch_chained(append_token_batched_kernel<T2>, dim3((unsigned)kv_heads, (unsigned)n_items), dim3(128), 0, st, true,
                                     dev, src_dtype), "append_token_batched_kernel");
}

// Appends the batch's tokens and leaves the records on the device.
int append_batched_launch(const cqa_batch_item *items, cqa_batch_item *dev, int n_items, int kv_heads, int t2_dtype, int src_dtype, cudaStream_t st)
{
    switch (t2_dtype) {
    case CQA_F32: return append_batched_t<float>(items, dev, n_items, kv_heads, src_dtype, st);
    case CQA_F16: return append_batched_t<__half>(items, dev, n_items, kv_heads, src_dtype, st);
    default: return append_batched_t<__nv_bfloat16>(items, dev, n_items, kv_heads, src_dtype, st);
    }
}

// Stand-alone per-token INT4 quantiser: one 8-thread group per token.
template <typename T>
__global__ void __launch_bounds__(128) int4_quantise_kernel(const T *x, long T_rows, uint8_t *packed,
                                                           uint16_t *scales, uint16_t *zeros,
                                                           float *rel_err, float *abs_err)
{
    const long t = (long)blockIdx.x * 16 + (threadIdx.x >> 3);
    const int g = threadIdx.x & 7;
    const bool live = t < T_rows;
    float xv[16];
    if (live) {
        float a[8], b[8];
        load8<T>(x + t * D + g * GS, a);
        load8<T>(x + t * D + g * GS + 8, b);
#pragma unroll
        for (int i = 0; i < 8; ++i) { xv[i] = a[i]; xv[i + 8] = b[i]; }
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) xv[i] = 0.0f;
    }
    uint2 pk;
    float s, z, da, db, xa, xb;
    int4_group(xv, pk, s, z, da, db);
    sumsq16(xv, xa, xb);
    float ae = __fsqrt_rn(group8_sum(da, db));
    float xn = fmaxf(__fsqrt_rn(group8_sum(xa, xb)), 1e-6f);
    if (live) {
        *reinterpret_cast<uint2 *>(packed + t * (D / 2) + g * 8) = pk;
        scales[t * NG + g] = __half_as_ushort(__float2half_rn(s));
        zeros[t * NG + g] = __half_as_ushort(__float2half_rn(z));
        if (g == 0) {
            if (rel_err) rel_err[t] = __fdiv_rn(ae, xn);
            if (abs_err) abs_err[t] = ae;
        }
    }
}

// ------------------------------------------------------------------ launchers

static int valid_cache(const cqa_cache *c)
{
    if (!c || !c->keys_int8 || !c->keys_scale || !c->keys_zero_points) {
        set_error("cqa_cache: NULL key arrays");
        return CQA_ERR_INVALID;
    }
    if (c->kv_heads <= 0 || c->cap_tokens <= 0 || c->max_blocks <= 0) {
        set_error("cqa_cache: bad sizes kv=%d cap=%ld max_blocks=%ld", c->kv_heads, (long)c->cap_tokens,
                  (long)c->max_blocks);
        return CQA_ERR_INVALID;
    }
    if (c->gqa_group != 1 && c->gqa_group != 2 && c->gqa_group != 4 && c->gqa_group != 8) {
        set_error("cqa_cache: gqa_group must be 1, 2, 4 or 8 (got %d)", c->gqa_group);
        return CQA_ERR_UNSUPPORTED;
    }
    return CQA_OK;
}

// The block encoder writes by bulk copies, which start on 16-byte boundaries (the score and attend kernels ask the
// same of these arrays).
static int encode_alignment(const cqa_cache *c)
{
    if (((uintptr_t)c->keys_int8 | (uintptr_t)c->keys_scale | (uintptr_t)c->keys_zero_points | (uintptr_t)c->values_int4_packed |
         (uintptr_t)c->values_int4_scales | (uintptr_t)c->values_int4_zeros | (uintptr_t)c->keys_t2 | (uintptr_t)c->values_t2 |
         (uintptr_t)c->keys_t2_backing | (uintptr_t)c->values_t2_backing) & 15) {
        set_error("cqa_cache: the key, INT4 value and Tier-2 arrays must be 16-byte aligned");
        return CQA_ERR_INVALID;
    }
    return CQA_OK;
}

// `chained`: the launch before it on the stream belongs to the same prefill (its kernel touches other memory and is
// waited for at the end of this one).
template <typename T>
static int launch_quantize(const cqa_cache *c, const void *k, const void *v, long src_rows, long first,
                           long n, cudaStream_t st, bool chained)
{
    const T *ks = reinterpret_cast<const T *>(k), *vs = reinterpret_cast<const T *>(v);
    int copy = 1;
    if (!c->key_slots && !c->value_slots && k == c->keys_t2 && v == c->values_t2 && src_rows == c->keys_t2_rows &&
        first == 0)
        copy = 0;
    // one wave of the resident CTAs where the prompt is long enough, at most 32 blocks per warp
    using LY = EncLayout<T>;
    static size_t granted[SMEM_ATTR_DEVICES] = {};
    const int rc = check_cuda(ensure_dynamic_smem(encode_blocks_kernel<T>, (size_t)LY::TOTAL, granted),
                              "cudaFuncSetAttribute(encode_blocks_kernel)");
    if (rc) return rc;
    const long warps = 148L * LY::CTAS * ENC_WARPS;
    long bpw = (n * c->kv_heads + warps - 1) / warps;
    bpw = bpw < 1 ? 1 : (bpw > 32 ? 32 : bpw);
    dim3 grid((unsigned)((n + ENC_WARPS * bpw - 1) / (ENC_WARPS * bpw)), (unsigned)c->kv_heads);
    return check_cuda(launch_chained(encode_blocks_kernel<T>, grid, dim3(ENC_WARPS * 32), LY::TOTAL, st, chained, *c, ks, vs,
                                     src_rows, first, n, (int)bpw, copy), "encode_blocks_kernel");
}

static int launch_quantize_any(const cqa_cache *c, const void *k, const void *v, int dtype, long src_rows, long first, long n,
                               cudaStream_t st, bool chained)
{
    switch (dtype) {
    case CQA_F32: return launch_quantize<float>(c, k, v, src_rows, first, n, st, chained);
    case CQA_F16: return launch_quantize<__half>(c, k, v, src_rows, first, n, st, chained);
    default: return launch_quantize<__nv_bfloat16>(c, k, v, src_rows, first, n, st, chained);
    }
}

template <typename T>
static int launch_tail(const cqa_prefill_item &it, long first_pos, int n_tail, cudaStream_t st, bool chained)
{
    dim3 grid(1u + (it.init_reserve ? TAIL_INIT_CTAS : 0), (unsigned)it.cache.kv_heads);
    return check_cuda(launch_chained(prefill_tail_kernel<T>, grid, dim3(256), 0, st, chained, it.cache,
                                     reinterpret_cast<const T *>(it.k_src), reinterpret_cast<const T *>(it.v_src),
                                     (long)it.src_rows, first_pos, n_tail, (int)it.defer_int4, (int)it.init_reserve),
                      "prefill_tail_kernel");
}

}  // namespace cqa

using namespace cqa;

int cqa::quantize_wait_timeouts(int *count, int reset) { return wait_timeouts_of_this_unit(count, reset); }

extern "C" int cqa_quantize_blocks(const cqa_cache *c, const void *k_src, const void *v_src, int src_dtype,
                                   int64_t src_rows, int64_t first_block, int64_t n_blocks, void *stream)
{
    int rc = valid_cache(c);
    if (rc) return rc;
    if (!k_src || !v_src) { set_error("cqa_quantize_blocks: NULL source"); return CQA_ERR_INVALID; }
    rc = encode_alignment(c);
    if (rc) return rc;
    if (n_blocks == 0) return CQA_OK;
    if (n_blocks < 0 || first_block < 0 || first_block + n_blocks > c->max_blocks ||
        (first_block + n_blocks) * BS > c->cap_tokens || n_blocks * BS > src_rows) {
        set_error("cqa_quantize_blocks: block range [%ld,+%ld) out of bounds", (long)first_block,
                  (long)n_blocks);
        return CQA_ERR_INVALID;
    }
    if ((c->keys_t2 || c->values_t2) && src_dtype != c->t2_dtype) {
        set_error("cqa_quantize_blocks: source dtype %d must equal the cache's Tier-2 dtype %d", src_dtype,
                  c->t2_dtype);
        return CQA_ERR_UNSUPPORTED;
    }
    if (src_dtype < 0 || src_dtype > 2) { set_error("cqa_quantize_blocks: unknown dtype %d", src_dtype); return CQA_ERR_INVALID; }
    return launch_quantize_any(c, k_src, v_src, src_dtype, src_rows, first_block, n_blocks, (cudaStream_t)stream, false);
}

// Argument checks of the append (shared with the batched step).
int cqa::append_check(const cqa_cache *c, const void *k_new, const void *v_new, int src_dtype, long pos)
{
    int rc = valid_cache(c);
    if (rc) return rc;
    if (!k_new || !v_new) { set_error("cqa_append_token: NULL token"); return CQA_ERR_INVALID; }
    if (pos < 0 || pos >= c->cap_tokens || pos / BS >= c->max_blocks) {
        set_error("cqa_append_token: position %ld beyond capacity %ld", pos, (long)c->cap_tokens);
        return CQA_ERR_TOO_LARGE;
    }
    if (src_dtype < 0 || src_dtype > 2) { set_error("cqa_append_token: unknown dtype"); return CQA_ERR_INVALID; }
    if (c->t2_dtype < 0 || c->t2_dtype > 2) { set_error("cqa_append_token: unknown Tier-2 dtype %d", c->t2_dtype); return CQA_ERR_INVALID; }
    return CQA_OK;
}

extern "C" int cqa_append_token(const cqa_cache *c, const void *k_new, const void *v_new, int src_dtype,
                                int64_t pos, int defer_int4, void *stream)
{
    int rc = append_check(c, k_new, v_new, src_dtype, pos);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    switch (c->t2_dtype) {
    case CQA_F32: rc = check_cuda(launch_chained(append_token_kernel<float>, dim3(c->kv_heads), dim3(128), 0, st, true, *c, k_new, v_new, src_dtype, pos, defer_int4), "append_token_kernel"); break;
    case CQA_F16: rc = check_cuda(launch_chained(append_token_kernel<__half>, dim3(c->kv_heads), dim3(128), 0, st, true, *c, k_new, v_new, src_dtype, pos, defer_int4), "append_token_kernel"); break;
    case CQA_BF16: rc = check_cuda(launch_chained(append_token_kernel<__nv_bfloat16>, dim3(c->kv_heads), dim3(128), 0, st, true, *c, k_new, v_new, src_dtype, pos, defer_int4), "append_token_kernel"); break;
    default: set_error("cqa_append_token: unknown Tier-2 dtype %d", c->t2_dtype); return CQA_ERR_INVALID;
    }
    return rc;
}

extern "C" int cqa_prefill_encode(const cqa_prefill_item *items, int n_items, int src_dtype, void *stream)
{
    if (!items || n_items <= 0) { set_error("cqa_prefill_encode: no items"); return CQA_ERR_INVALID; }
    if (src_dtype < 0 || src_dtype > 2) { set_error("cqa_prefill_encode: unknown dtype %d", src_dtype); return CQA_ERR_INVALID; }
    // every check before the first launch
    for (int i = 0; i < n_items; ++i) {
        const cqa_prefill_item &it = items[i];
        int rc = valid_cache(&it.cache);
        if (!rc) rc = encode_alignment(&it.cache);
        if (rc) return rc;
        if (!it.k_src || !it.v_src || it.n_tokens < 0 || it.src_rows < it.n_tokens) {
            set_error("cqa_prefill_encode: item %d: bad source (%ld tokens in %ld rows)", i, (long)it.n_tokens, (long)it.src_rows);
            return CQA_ERR_INVALID;
        }
        const long nblk = (it.n_tokens + BS - 1) / BS;
        if (it.n_tokens > it.cache.cap_tokens || nblk > it.cache.max_blocks) {
            set_error("cqa_prefill_encode: item %d: %ld tokens exceed the cache capacity %ld", i, (long)it.n_tokens,
                      (long)it.cache.cap_tokens);
            return CQA_ERR_TOO_LARGE;
        }
        if ((it.cache.keys_t2 || it.cache.values_t2) && src_dtype != it.cache.t2_dtype) {
            set_error("cqa_prefill_encode: item %d: source dtype %d must equal the cache's Tier-2 dtype %d", i, src_dtype,
                      it.cache.t2_dtype);
            return CQA_ERR_UNSUPPORTED;
        }
    }
    cudaStream_t st = (cudaStream_t)stream;
    bool chained = false;   // the first launch follows whatever wrote the prompt
    for (int i = 0; i < n_items; ++i) {
        const cqa_prefill_item &it = items[i];
        const long full = it.n_tokens / BS;
        const int tail = (int)(it.n_tokens - full * BS);
        int rc = CQA_OK;
        if (full > 0) {
            rc = launch_quantize_any(&it.cache, it.k_src, it.v_src, src_dtype, it.src_rows, 0, full, st, chained);
            if (rc) return rc;
            chained = true;
        }
        if (tail > 0 || it.init_reserve) {
            switch (src_dtype) {
            case CQA_F32: rc = launch_tail<float>(it, full * BS, tail, st, chained); break;
            case CQA_F16: rc = launch_tail<__half>(it, full * BS, tail, st, chained); break;
            default: rc = launch_tail<__nv_bfloat16>(it, full * BS, tail, st, chained); break;
            }
            if (rc) return rc;
            chained = true;
        }
    }
    return CQA_OK;
}

extern "C" int cqa_int4_quantise(const void *x, int src_dtype, int64_t T, uint8_t *packed, uint16_t *scales,
                                 uint16_t *zeros, float *rel_err, float *abs_err, void *stream)
{
    if (!x || !packed || !scales || !zeros) { set_error("cqa_int4_quantise: NULL pointer"); return CQA_ERR_INVALID; }
    if (T == 0) return CQA_OK;
    if (T < 0) { set_error("cqa_int4_quantise: negative row count"); return CQA_ERR_INVALID; }
    cudaStream_t st = (cudaStream_t)stream;
    unsigned grid = (unsigned)((T + 15) / 16);
    switch (src_dtype) {
    case CQA_F32: int4_quantise_kernel<float><<<grid, 128, 0, st>>>((const float *)x, T, packed, scales, zeros, rel_err, abs_err); note_launch(); break;
    case CQA_F16: int4_quantise_kernel<__half><<<grid, 128, 0, st>>>((const __half *)x, T, packed, scales, zeros, rel_err, abs_err); note_launch(); break;
    case CQA_BF16: int4_quantise_kernel<__nv_bfloat16><<<grid, 128, 0, st>>>((const __nv_bfloat16 *)x, T, packed, scales, zeros, rel_err, abs_err); note_launch(); break;
    default: set_error("cqa_int4_quantise: unknown dtype %d", src_dtype); return CQA_ERR_INVALID;
    }
    return check_launch("int4_quantise_kernel");
}
