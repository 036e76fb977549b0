// Phase 2: mixed INT8/FP16-key, INT4/FP16-value split-K attend, the dense
// FP16 recompute of flagged heads, and the log-sum-exp merge — one launch.
//
// attend_kernel, grid (splits, KV * groups of at most four heads):
//   * A CTA takes one (KV head, group of heads, split of blocks), a warp one pair of neighbouring 16-token blocks at a
//     time; their INT4 codes, scales, zeros and cached Phase-1 token scores arrive in a warp-private two-stage
//     shared-memory ring through 16-byte asynchronous copies, so no CTA barrier sits in the loop.  (Three stages
//     measured the same.)  Softmax weights are made in the layout of the matrix products' B fragments.
//   * (head, block) pairs flagged in topk_mask take their logits from Tier-2 keys, pairs flagged in value_mask their
//     values from Tier 2: the same products, the four heads together.  The rows are requested into L2 two pairs ahead.
//   * Heads that the certificate flags for the dense FP16 recompute: when a CTA is done with its split it draws units
//     of (group with a flagged head, chunk of blocks) from a counter; CTAs beyond the splits, where the GPU has room for
//     them, start there.  With no flagged head this is one word read.
//   * The last CTA to finish for a KV head (a group, for the dense part) merges the split partials and writes the
//     output rows; no separate merge launch.
//
// Bound: instruction issue (about 400 warp instructions per block and four heads, 0.57 issued per cycle and
// scheduler) and the latency of the promoted rows; HBM (96 bytes per token and KV head and 256 per promoted row) is at
// 33 %.  131072 tokens x 8 KV heads x 4, bf16, 64 planted blocks: 73 us as packed float32 multiply-adds on the CUDA
// cores with one pass per promoted head, 55 us so; 100003 tokens, eight heads per KV head, diffuse: 292 -> 191 us.
//
// Nothing computed here can change a selection or a certificate flag, so fast exponentials are used.
#include <mutex>
#include <type_traits>

#include "common.cuh"

namespace cqa {

constexpr int ATT_WARPS = 8;
constexpr int ATT_THREADS = ATT_WARPS * 32;
constexpr int ATT_STAGES = 2;

// exp(x) by the exponential unit; results below 2^-126 are zero (the subnormal range costs four instructions a call).
__device__ __forceinline__ float fexp(float x)
{
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x * 1.4426950408889634f));
    return r;
}

__device__ __forceinline__ void att_cp16(void *smem, const void *gmem)
{
    unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void att_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void att_wait()
{
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// ---------------------------------------------------------------- tensor-core pieces of a block
//
// A block is a contraction of 16 tokens: values^T [channels x 16 tokens] times weights [16 tokens x columns], as
// m16n8k16 products with float32 accumulators.  (The 16-token blocks, four heads and per-token scales make the
// operands far smaller than the tiles the tcgen05 unit works on; 17 instructions per block of this shape keep the
// tensor pipe 20 % busy.)  Nothing is rounded away: a float32 weight enters
// as two fp16 pieces (22 bits, half an ulp of float32) or three bf16 pieces (24 bits), codes and Tier-2 values enter
// exactly.
//
// INT4 codes: one ldmatrix.trans hands lane (r = lane / 4, q = lane % 4) the 16-bit word r of a 32-channel chunk for
// tokens 2q and 2q + 1, i.e. the codes of channels 4r..4r+3; a logic operation and a packed half operation turn two of
// them into matrix elements.  Tile (chunk c, j) has rows r <-> channel 32c + 4r + j and r + 8 <-> channel + 2.  Rows
// 0-3 belong to value group 2c, rows 4-7 to group 2c + 1, and the scales differ between the two, so the columns are
// (head h, parity p): column h + 4p carries weight * scale of group 2c + p and is used for the rows of that parity
// only (half of each tile is not used; the tensor pipe has room).
//
// The tensor core truncates its sums (a chain of n products loses n * 2^-24 in one direction: 3e-5 over 256 blocks),
// so a block's products start from zero, lower pieces first, and are added to the accumulators by rounded float32
// additions; the error is then that of a chain of float32 fused multiply-adds (2e-7 to 5e-7 of the result).  Codes enter as code - 8 and the
// zero points as zero + 8 * scale (the middle of the group's range; one small product per block, rows 0-7 its upper and
// rows 8-15 its lower fp16 piece), which keeps the terms at the size of the result.
__device__ __forceinline__ void mma_f16(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <bool BF16>
__device__ __forceinline__ void mma_first(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1)
{
    if (BF16)
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                     : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                     : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
    else
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                     : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                     : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
}
__device__ __forceinline__ void add4(float (&acc)[4], const float (&d)[4])
{
    const float2 x = __fadd2_rn(make_float2(acc[0], acc[1]), make_float2(d[0], d[1]));
    const float2 y = __fadd2_rn(make_float2(acc[2], acc[3]), make_float2(d[2], d[3]));
    acc[0] = x.x; acc[1] = x.y; acc[2] = y.x; acc[3] = y.y;
}
__device__ __forceinline__ void ldmatrix_x4_trans(unsigned (&x)[4], unsigned addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix_x2_trans(unsigned &x0, unsigned &x1, unsigned addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(x0), "=r"(x1) : "r"(addr) : "memory");
}
__device__ __forceinline__ unsigned as_u32(__half2 v) { return *reinterpret_cast<unsigned *>(&v); }
__device__ __forceinline__ __half2 as_half2(unsigned v) { return *reinterpret_cast<__half2 *>(&v); }
// x = hi + lo to half an ulp of float32, two values at a time (fp16 pieces; |x| within the normal range of fp16).
__device__ __forceinline__ void split_f16(float2 x, unsigned &hi, unsigned &lo)
{
    const __half2 h = __float22half2_rn(x);
    const float2 back = __half22float2(h);
    hi = as_u32(h);
    lo = as_u32(__float22half2_rn(__ffma2_rn(back, make_float2(-1.0f, -1.0f), x)));
}
// x = hi + mid + lo exactly (bf16 pieces of 8 bits each).
__device__ __forceinline__ unsigned pack_bf16(float2 x)
{
    const __nv_bfloat162 b = __float22bfloat162_rn(x);
    return *reinterpret_cast<const unsigned *>(&b);
}
__device__ __forceinline__ float2 unpack_bf16(unsigned w) { return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }
__device__ __forceinline__ void split_bf16(float2 x, unsigned &hi, unsigned &mid, unsigned &lo)
{
    hi = pack_bf16(x);
    x = __ffma2_rn(unpack_bf16(hi), make_float2(-1.0f, -1.0f), x);
    mid = pack_bf16(x);
    x = __ffma2_rn(unpack_bf16(mid), make_float2(-1.0f, -1.0f), x);
    lo = pack_bf16(x);
}
// (a & b) | c in one logic instruction.
__device__ __forceinline__ unsigned and_or(unsigned a, unsigned b, unsigned c)
{
    unsigned d;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

template <int G, typename T2>
struct AttLayout {
    static constexpr int HG = G > 4 ? 4 : G;                  // heads a CTA works on
    static constexpr int SUBS = G / HG;                       // CTAs per (KV head, split)
    // a stage holds two neighbouring blocks, each array for both: codes (chunk c of token t at t * 64 +
    // 16 * (c ^ ((t >> 1) & 3))), scales, zeros, token scores [4][16]
    static constexpr int PACKED = 0, PACKED_BLK = BS * (D / 2);
    static constexpr int SCALES = PACKED + 2 * PACKED_BLK, SCALES_BLK = BS * NG * 2;
    static constexpr int ZEROS = SCALES + 2 * SCALES_BLK;
    static constexpr int SCORES = ZEROS + 2 * SCALES_BLK, SCORES_BLK = 4 * BS * 4;
    static constexpr int STAGE = SCORES + 2 * SCORES_BLK;
    static constexpr int RING = ATT_WARPS * ATT_STAGES * STAGE;
    // cross-warp merge buffers and final-merge scratch (both alias the ring)
    static constexpr int MERGE_A = ATT_WARPS * HG * (D + 2) * 4;
    static constexpr int MERGE_SPLITS = CQA_MAX_SPLITS > CQA_MAX_DENSE_SPLITS ? CQA_MAX_SPLITS : CQA_MAX_DENSE_SPLITS;
    static constexpr int MERGE_B = (ATT_WARPS * MERGE_SPLITS + ATT_WARPS + ATT_WARPS * D) * 4;
    static constexpr int MERGE = MERGE_A > MERGE_B ? MERGE_A : MERGE_B;
    static constexpr int RING_BYTES = RING > MERGE ? RING : MERGE;
    // the query as matrix fragments: [pieces 0,1 | piece 2][8 steps][32 lanes] words of two 16-bit pairs; with float32
    // Tier-2 rows the query rows themselves, and a weight tile per warp
    static constexpr bool F32 = std::is_same<T2, float>::value;
    static constexpr int QFRAG = F32 ? HG * D * 4 : 2 * 8 * 32 * 8;
    static constexpr int WTILE = F32 ? BS * 4 * 4 : 0;        // [16 tokens][4 heads]
    static constexpr int TOTAL = RING_BYTES + QFRAG + ATT_WARPS * WTILE;
};

// Per-lane source pointers of the next unit (block or pair of blocks) to stage.
template <int G, typename T2>
struct AttIssuer {
    using LY = AttLayout<G, T2>;
    const char *pk, *s, *z, *sc;   // global sources for this lane
    int b, b_end;                  // first block of the unit to issue next
    int unit;                      // blocks of a unit: 1 or 2
    int at;                        // swizzled place of this lane's 16 code bytes within 512
    bool have4;

    __device__ __forceinline__ void init(const cqa_cache &c, const float *tok, int nq_, int kv, int sub, int b0, int bend, int unit_,
                                         int lane)
    {
        b = b0;
        b_end = min(bend, nq_);
        unit = unit_;
        have4 = c.values_int4_packed != nullptr;
        const int t = lane >> 2;
        at = t * 64 + 16 * ((lane & 3) ^ ((t >> 1) & 3));      // eight tokens per round, the same pattern in each
        const long row0 = (long)kv * c.cap_tokens + (long)b0 * BS;
        pk = reinterpret_cast<const char *>(c.values_int4_packed) + row0 * (D / 2) + lane * 16;
        s = reinterpret_cast<const char *>(c.values_int4_scales) + row0 * NG * 2 + lane * 16;
        z = reinterpret_cast<const char *>(c.values_int4_zeros) + row0 * NG * 2 + lane * 16;
        // lane = (block of the pair, head, 16 bytes)
        sc = reinterpret_cast<const char *>(tok + ((long)kv * nq_ + b0 + lane / (4 * LY::HG)) * G * BS + sub * LY::HG * BS) +
             (lane % (4 * LY::HG)) * 16;
    }
    // Stage the unit's blocks (as far as they are quantised blocks of this CTA) and advance by a warp stride; always
    // commits one group.
    __device__ __forceinline__ void issue(char *stage, int lane)
    {
        if (b < b_end) {
            const bool two = unit == 2 && b + 1 < b_end;
            if (have4) {
                att_cp16(stage + at, pk);
                att_cp16(stage + at + 512, pk + 512);
                if (two) {
                    att_cp16(stage + at + 1024, pk + 1024);
                    att_cp16(stage + at + 1536, pk + 1536);
                }
                if (two || lane < 16) {
                    att_cp16(stage + LY::SCALES + lane * 16, s);
                    att_cp16(stage + LY::ZEROS + lane * 16, z);
                }
            }
            if (lane < (two ? 8 : 4) * LY::HG) {
                const int blk = lane / (4 * LY::HG);
                att_cp16(stage + LY::SCORES + blk * LY::SCORES_BLK + (lane - blk * 4 * LY::HG) * 16, sc);
            }
        }
        att_commit();
        const int step = unit * ATT_WARPS;
        b += step;
        pk += step * (BS * (D / 2));
        s += step * (BS * NG * 2);
        z += step * (BS * NG * 2);
        sc += step * (G * BS * 4);
    }
};

// Running state of one warp over its blocks.  Lane (n = lane / 4, q = lane % 4): head h = n % 4, parity n / 4, tokens
// 2q, 2q + 1, 2q + 8, 2q + 9.
template <int G, typename T2>
struct AttWarp {
    using LY = AttLayout<G, T2>;
    static constexpr int HG = LY::HG;
    static constexpr bool F32 = LY::F32, F16 = std::is_same<T2, __half>::value;
    // Weights are multiplied by F, the largest power of two up to 2^15 that keeps weight * scale within fp16, and the
    // accumulators are scaled back at the end.
    float acc[8][4];        // tile 2c + j
    float zacc[4];          // middles of the groups: row = group (+ 8: lower piece), column = head + 4 * piece
    float2 facc[F32 ? 4 : 1][4];   // float32 Tier-2 values: lane L (mod 16) channels 8L.., half warps take even / odd tokens
    float m, l;             // running maximum of head h; this lane's share of the running sum
    float F;
    int lane, q, h, par;
    bool head_ok;           // h is a head of this group
    unsigned prmt_sel;

    __device__ __forceinline__ void init(int lane_, float m0, float F_)
    {
        lane = lane_;
        q = lane & 3;
        h = (lane >> 2) & 3;
        par = lane >> 4;
        head_ok = h < HG;
        prmt_sel = par ? 0x7632u : 0x5410u;
        m = head_ok ? m0 : 0.0f;
        l = 0.0f;
        F = F_;
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[i][k] = 0.0f;
#pragma unroll
        for (int k = 0; k < 4; ++k) zacc[k] = 0.0f;
        if (F32) {
#pragma unroll
            for (int g = 0; g < 4; ++g)
#pragma unroll
                for (int k = 0; k < 4; ++k) facc[F32 ? g : 0][k] = make_float2(0.0f, 0.0f);
        }
    }

    // FP16-key logits of the heads in `km` from the Tier-2 rows of a block, into sc[4][16]; tokens from n_valid on get
    // -infinity.
    __device__ __forceinline__ void key_logits(const T2 *kblk, unsigned km, int n_valid, float q_scale, const char *qfrag,
                                               bool third, float *sc)
    {
        if constexpr (F32) {
            const float *qrow = reinterpret_cast<const float *>(qfrag);
            const int L = lane & 15, hw = lane >> 4;
#pragma unroll 1
            for (int half = 0; half < 2; ++half) {
                Raw8<T2> kr[4];       // four rows in flight
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int t = hw * 8 + half * 4 + i;
                    kr[i] = (t < n_valid && kblk != nullptr) ? raw_load8<T2>(kblk + t * D + 8 * L) : raw_zero8<T2>();
                }
#pragma unroll 1
                for (int g = 0; g < HG; ++g) {
                    if (!(km & (1u << g))) continue;
                    float qv[8];
                    load8<float>(qrow + g * D + 8 * L, qv);
                    float p[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        float kf[8];
                        raw_to_f(kr[i], kf);
                        p[i] = chain8(kf, qv);
                    }
                    // sums over the 16 lanes of four rows at once: lane L ends with row i = L / 4
                    const bool u8 = (L & 8) != 0, u4 = (L & 4) != 0;
                    const float a0 = (u8 ? p[2] : p[0]) + __shfl_xor_sync(FULL, u8 ? p[0] : p[2], 8);
                    const float a1 = (u8 ? p[3] : p[1]) + __shfl_xor_sync(FULL, u8 ? p[1] : p[3], 8);
                    float d = (u4 ? a1 : a0) + __shfl_xor_sync(FULL, u4 ? a0 : a1, 4);
                    d += __shfl_xor_sync(FULL, d, 2);
                    d += __shfl_xor_sync(FULL, d, 1);
                    const int t = hw * 8 + half * 4 + (L >> 2);
                    if ((L & 3) == 0) sc[g * BS + t] = t < n_valid ? d * q_scale : -INFINITY;
                }
            }
        } else {
            // rows: tokens r and r + 8; lane q holds channels 32i + 8q .. + 7 of steps 2i and 2i + 1
            const int r = lane >> 2;
            uint4 a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
                a[i] = (r < n_valid && kblk) ? *reinterpret_cast<const uint4 *>(kblk + r * D + 32 * i + 8 * q) : zero;
                b[i] = (r + 8 < n_valid && kblk) ? *reinterpret_cast<const uint4 *>(kblk + (r + 8) * D + 32 * i + 8 * q) : zero;
            }
            float d[4], e[4][4];
            const uint2 *qf = reinterpret_cast<const uint2 *>(qfrag) + lane;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint2 q0 = qf[(2 * i) * 32], q1 = qf[(2 * i + 1) * 32];
                mma_first<!F16>(e[i], a[i].x, b[i].x, a[i].y, b[i].y, q0.x, q0.y);
                if constexpr (F16) {
                    mma_f16(e[i], a[i].z, b[i].z, a[i].w, b[i].w, q1.x, q1.y);
                } else {
                    mma_bf16(e[i], a[i].z, b[i].z, a[i].w, b[i].w, q1.x, q1.y);
                    if (third) {
                        const uint2 p0 = qf[(8 + 2 * i) * 32], p1 = qf[(9 + 2 * i) * 32];
                        mma_bf16(e[i], a[i].x, b[i].x, a[i].y, b[i].y, p0.x, p0.y);
                        mma_bf16(e[i], a[i].z, b[i].z, a[i].w, b[i].w, p1.x, p1.y);
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) d[k] = (e[0][k] + e[1][k]) + (e[2][k] + e[3][k]);
            // columns n and n + 4 hold the pieces of one head
#pragma unroll
            for (int k = 0; k < 4; ++k) d[k] += __shfl_xor_sync(FULL, d[k], 2);
            if (q < 2) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int g = 2 * q + (k & 1), t = r + 8 * (k >> 1);
                    if (km & (1u << g)) sc[g * BS + t] = t < n_valid ? d[k] * q_scale : -INFINITY;
                }
            }
        }
        __syncwarp();
    }

    // Softmax weights of this lane's four tokens from sc[4][16]; `move`: the running maximum may have to rise.
    __device__ __forceinline__ void weights(const float *sc, bool move, float2 &w0, float2 &w1)
    {
        float2 x0 = *reinterpret_cast<const float2 *>(sc + h * BS + 2 * q);
        float2 x1 = *reinterpret_cast<const float2 *>(sc + h * BS + 2 * q + 8);
        if (HG < 4 && !head_ok) x0 = x1 = make_float2(-INFINITY, -INFINITY);
        if (move) {
            float bm = fmaxf(fmaxf(x0.x, x0.y), fmaxf(x1.x, x1.y));
            bm = fmaxf(bm, __shfl_xor_sync(FULL, bm, 1));
            bm = fmaxf(bm, __shfl_xor_sync(FULL, bm, 2));
            const float up = fmaxf(m, bm);
            const float alpha = m == up ? 1.0f : fexp(m - up);     // 0 when there was no maximum yet
            m = up;
            if (__any_sync(FULL, alpha != 1.0f)) {
                l *= alpha;
                const float a0 = __shfl_sync(FULL, alpha, ((2 * q) & 3) * 4), a1 = __shfl_sync(FULL, alpha, ((2 * q + 1) & 3) * 4);
#pragma unroll
                for (int i = 0; i < 8; ++i) { acc[i][0] *= a0; acc[i][1] *= a1; acc[i][2] *= a0; acc[i][3] *= a1; }
                zacc[0] *= a0; zacc[1] *= a1; zacc[2] *= a0; zacc[3] *= a1;
                if (F32) {
#pragma unroll
                    for (int g = 0; g < HG; ++g) {
                        const float ag = __shfl_sync(FULL, alpha, g * 4);
#pragma unroll
                        for (int k = 0; k < 4; ++k) facc[F32 ? g : 0][k] = __fmul2_rn(facc[F32 ? g : 0][k], make_float2(ag, ag));
                    }
                }
            }
        }
        w0 = make_float2(fexp(x0.x - m), fexp(x0.y - m));
        w1 = make_float2(fexp(x1.x - m), fexp(x1.y - m));
        l += (w0.x + w0.y) + (w1.x + w1.y);
    }

    // INT4 values of a staged block; `on` = 0 for a head that reads Tier-2 values, else 1.  The weights are split into
    // fp16 pieces once; weight * scale comes out of packed half operations as the rounded product, and its exact
    // remainder plus the lower piece's product (22 bits in all).
    __device__ __forceinline__ void int4_values(unsigned codes, const char *scales, unsigned scales_a, unsigned zeros_a, float on,
                                                float2 w0, float2 w1)
    {
        unsigned hi0, lo0, hi1, lo1;
        const float f = on * F;
        split_f16(__fmul2_rn(w0, make_float2(f, f)), hi0, lo0);
        split_f16(__fmul2_rn(w1, make_float2(f, f)), hi1, lo1);
        const int t = lane & 15;
        {
            // zero and scale of group lane / 4 for this lane's tokens
            unsigned z0, z1, s0, s1, mh0, ml0, mh1, ml1;
            ldmatrix_x2_trans(z0, z1, zeros_a + t * 16);
            ldmatrix_x2_trans(s0, s1, scales_a + t * 16);
            const float2 eight = make_float2(8.0f, 8.0f);
            split_f16(__ffma2_rn(__half22float2(as_half2(s0)), eight, __half22float2(as_half2(z0))), mh0, ml0);
            split_f16(__ffma2_rn(__half22float2(as_half2(s1)), eight, __half22float2(as_half2(z1))), mh1, ml1);
            float d[4];
            mma_first<false>(d, mh0, ml0, mh1, ml1, par ? lo0 : hi0, par ? lo1 : hi1);
            add4(zacc, d);
        }
        const uint4 *srow = reinterpret_cast<const uint4 *>(scales);
        const uint4 sa = srow[2 * q], sb = srow[2 * q + 1], sc_ = srow[2 * q + 8], sd = srow[2 * q + 9];
        const unsigned *pa = &sa.x, *pb = &sb.x, *pc = &sc_.x, *pd = &sd.x;
        const auto scaled = [](unsigned hi, unsigned lo, unsigned sc2, unsigned &ph, unsigned &pl) {
            const __half2 h2 = as_half2(hi), s2 = as_half2(sc2);
            const __half2 p = __hmul2_rn(h2, s2);
            ph = as_u32(p);
            pl = as_u32(__hfma2(as_half2(lo), s2, __hfma2(h2, s2, __hneg2(p))));
        };
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
            // matrices: tokens 0-7 and 8-15 of chunk 2cc, then of chunk 2cc + 1
            unsigned x[4];
            const int c = 2 * cc + (lane >> 4);
            ldmatrix_x4_trans(x, codes + t * 64 + 16 * (c ^ ((t >> 1) & 3)));
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int ch = 2 * cc + k;
                unsigned h0, l0, h1, l1;
                scaled(hi0, lo0, __byte_perm(pa[ch], pb[ch], prmt_sel), h0, l0);
                scaled(hi1, lo1, __byte_perm(pc[ch], pd[ch], prmt_sel), h1, l1);
                const unsigned a = x[2 * k], b = x[2 * k + 1], a8 = a >> 8, b8 = b >> 8;
                // code - 8: 1024 + code and 1024 + 16 code are exact half patterns
                const __half2 off0 = __float2half2_rn(-1032.0f), off1 = __float2half2_rn(-72.0f), sixteenth = __float2half2_rn(0.0625f);
                const unsigned M = 0x64006400u;
                const auto lo4 = [&](unsigned v) { return as_u32(__hadd2(as_half2(and_or(v, 0x000F000Fu, M)), off0)); };
                const auto hi4 = [&](unsigned v) { return as_u32(__hfma2(as_half2(and_or(v, 0x00F000F0u, M)), sixteenth, off1)); };
                unsigned p0 = lo4(a), p1 = lo4(a8), p2 = lo4(b), p3 = lo4(b8);
                float d[4], e[4];
                mma_first<false>(d, p0, p1, p2, p3, l0, l1);
                mma_f16(d, p0, p1, p2, p3, h0, h1);
                p0 = hi4(a); p1 = hi4(a8); p2 = hi4(b); p3 = hi4(b8);
                mma_first<false>(e, p0, p1, p2, p3, l0, l1);
                mma_f16(e, p0, p1, p2, p3, h0, h1);
                add4(acc[2 * ch], d);
                add4(acc[2 * ch + 1], e);
            }
        }
    }

    // Tier-2 values of a block for the heads in `vm` (weights of the others are zero).  Two-byte rows: lane (r, q)
    // holds tokens 2q, 2q + 1, 2q + 8, 2q + 9 and the channels 32c + 4r .. + 3 that the INT4 tiles give the same rows.
    __device__ __forceinline__ void t2_values(const T2 *vblk, unsigned vm, int n_valid, float2 w0, float2 w1, float *wtile)
    {
        if constexpr (F32) {
            if (par == 0) {
                wtile[(2 * q) * 4 + h] = w0.x;
                wtile[(2 * q + 1) * 4 + h] = w0.y;
                wtile[(2 * q + 8) * 4 + h] = w1.x;
                wtile[(2 * q + 9) * 4 + h] = w1.y;
            }
            __syncwarp();
            const int L = lane & 15, hw = lane >> 4;
#pragma unroll 1
            for (int half = 0; half < 2; ++half) {
                Raw8<T2> vr[4];       // four rows in flight
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int t = 8 * half + 2 * i + hw;
                    vr[i] = (t < n_valid && vblk != nullptr) ? raw_load8<T2>(vblk + t * D + 8 * L) : raw_zero8<T2>();
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int t = 8 * half + 2 * i + hw;
                    float v[8];
                    raw_to_f(vr[i], v);
                    const float4 w = *reinterpret_cast<const float4 *>(wtile + t * 4);
                    const float wg[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                    for (int g = 0; g < HG; ++g) {
                        if (!(vm & (1u << g))) continue;
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            facc[F32 ? g : 0][k] = __ffma2_rn(make_float2(wg[g], wg[g]), make_float2(v[2 * k], v[2 * k + 1]), facc[F32 ? g : 0][k]);
                    }
                }
            }
            __syncwarp();
        } else {
            const int r = lane >> 2;
            const float s = ((vm >> h) & 1u) ? F : 0.0f;
            w0 = __fmul2_rn(w0, make_float2(s, s));
            w1 = __fmul2_rn(w1, make_float2(s, s));
            unsigned p0[3], p1[3];
            if constexpr (F16) {
                split_f16(w0, p0[0], p0[1]);
                split_f16(w1, p1[0], p1[1]);
            } else {
                split_bf16(w0, p0[0], p0[1], p0[2]);
                split_bf16(w1, p1[0], p1[1], p1[2]);
            }
            {
                uint2 v[4][4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int t = 2 * q + (k & 1) + 8 * (k >> 1);
                    const bool ok = t < n_valid && vblk != nullptr;
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        v[k][c] = ok ? *reinterpret_cast<const uint2 *>(vblk + t * D + 32 * c + 4 * r) : make_uint2(0u, 0u);
                }
#pragma unroll
                for (int c = 0; c < 4; ++c) {
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const unsigned sel = j ? 0x7632u : 0x5410u;
                        const unsigned a0 = __byte_perm(v[0][c].x, v[1][c].x, sel), a1 = __byte_perm(v[0][c].y, v[1][c].y, sel);
                        const unsigned a2 = __byte_perm(v[2][c].x, v[3][c].x, sel), a3 = __byte_perm(v[2][c].y, v[3][c].y, sel);
                        float d[4];
                        if constexpr (F16) {
                            mma_first<false>(d, a0, a1, a2, a3, p0[1], p1[1]);
                            mma_f16(d, a0, a1, a2, a3, p0[0], p1[0]);
                        } else {
                            mma_first<true>(d, a0, a1, a2, a3, p0[2], p1[2]);
                            mma_bf16(d, a0, a1, a2, a3, p0[1], p1[1]);
                            mma_bf16(d, a0, a1, a2, a3, p0[0], p1[0]);
                        }
                        add4(acc[2 * c + j], d);
                    }
                }
            }
        }
    }

    // This warp's (max, sum, acc[128]) of every head into the CTA's merge buffers.
    __device__ __forceinline__ void store(float *sm_m, float *sm_l, float *sm_acc, int warp)
    {
        l += __shfl_xor_sync(FULL, l, 1);
        l += __shfl_xor_sync(FULL, l, 2);
        if (par == 0 && q == 0 && head_ok) { sm_m[warp * HG + h] = m; sm_l[warp * HG + h] = l; }
        float z0 = zacc[0] + zacc[2], z1 = zacc[1] + zacc[3];
        z0 += __shfl_xor_sync(FULL, z0, 2);
        z1 += __shfl_xor_sync(FULL, z1, 2);
        const float inv = 1.0f / F;
        const int r = lane >> 2, hA = 2 * (q & 1);
        const bool mine = (q >> 1) == (r >> 2);        // the columns of these rows' parity
        float *row = sm_acc + warp * HG * D;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int src = (2 * c + (r >> 2)) * 4 + (q & 1);
            const float za = __shfl_sync(FULL, z0, src) * inv, zb = __shfl_sync(FULL, z1, src) * inv;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int ch = 32 * c + 4 * r + j;
                if (mine && hA < HG) {
                    row[hA * D + ch] = fmaf(acc[2 * c + j][0], inv, za);
                    row[hA * D + ch + 2] = fmaf(acc[2 * c + j][2], inv, za);
                }
                if (mine && hA + 1 < HG) {
                    row[(hA + 1) * D + ch] = fmaf(acc[2 * c + j][1], inv, zb);
                    row[(hA + 1) * D + ch + 2] = fmaf(acc[2 * c + j][3], inv, zb);
                }
            }
        }
        if constexpr (F32) {
            __syncwarp();
            const int L = lane & 15;
#pragma unroll
            for (int g = 0; g < HG; ++g)
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float a = facc[g][k].x + __shfl_xor_sync(FULL, facc[g][k].x, 16), b = facc[g][k].y + __shfl_xor_sync(FULL, facc[g][k].y, 16);
                    if (lane < 16) { row[g * D + 8 * L + 2 * k] += a; row[g * D + 8 * L + 2 * k + 1] += b; }
                }
        }
    }
};

// Cross-warp merge of the buffers AttWarp::store filled: one partial per head to global memory.
template <int HG>
__device__ __forceinline__ void cta_merge_store(const float *sm_m, const float *sm_l, const float *sm_acc, float *out_m,
                                                float *out_l, float *out_acc, int head0, int split, int nsplits)
{
    __syncthreads();
    for (int item = threadIdx.x; item < HG * D; item += ATT_THREADS) {
        const int g = item / D, ch = item % D;
        float M = -INFINITY;
#pragma unroll
        for (int w = 0; w < ATT_WARPS; ++w) M = fmaxf(M, sm_m[w * HG + g]);
        float a = 0.0f, ll = 0.0f;
#pragma unroll
        for (int w = 0; w < ATT_WARPS; ++w) {
            const float mw = sm_m[w * HG + g];
            const float sc = mw == -INFINITY ? 0.0f : fexp(mw - M);
            a = fmaf(sm_acc[(w * HG + g) * D + ch], sc, a);
            ll = fmaf(sm_l[w * HG + g], sc, ll);
        }
        const long p = (long)(head0 + g) * nsplits + split;
        out_acc[p * D + ch] = a;
        if (ch == 0) { out_m[p] = M; out_l[p] = ll; }
    }
}

// Final merge of `ns` split partials of heads [head0, head0+nh) by the last CTA to arrive; bit i of `flagged`: head
// head0 + i is recomputed densely.  All 256 threads take part; `sm` is 16-byte aligned scratch of at least
// 8 * ns + 8 + 8*128 floats that no thread uses any more.
// A thread owns one float4 column of one head and every (256 / (32*nh))-th split.  Its accumulator rows are
// requested first (up to 20 loads in flight per thread) together with the (m, l) partials, which every warp turns into
// the per-split scales of its head by itself; the rows are then scaled and summed, the per-thread sums combined
// through shared memory, normalised and written.  (A chain of latencies, about 2 us; with the scales made by one warp
// per head between two CTA barriers and the flags read at the end, it and the ticket took 5 us of a 12 us kernel at
// 8192 tokens.)
__device__ __forceinline__ void final_merge(const float *pm, const float *pl, const float *pa, int ns, int head0,
                                            int nh, const cqa_workspace &ws, bool dense_role, unsigned flagged, float *sm, int kv_heads,
                                            int n_heads_total, int arrivals = 1)
{
    constexpr int BATCH = 20;
    const bool push_c = ws.partial_out != nullptr && ws.peer_world > 0 && ws.peer_partial[0] != nullptr;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float *s_sc = sm + warp * ns, *s_part = sm + ((ATT_WARPS * ns + 3) & ~3), *s_l = s_part + ATT_WARPS * D;
    const int nparts = ATT_WARPS / nh;      // nh is 1, 2, 4 or 8
    const int g = warp / nparts, part = warp % nparts;
    const float *gm = pm + (long)(head0 + g) * ns, *gl = pl + (long)(head0 + g) * ns;
    const float4 *rows = reinterpret_cast<const float4 *>(pa + (long)(head0 + g) * ns * D) + lane;
    float4 buf[BATCH];
    const auto load_rows = [&](int first) {
#pragma unroll
        for (int j = 0; j < BATCH; ++j) {
            const int sp = first + part + j * nparts;
            buf[j] = sp < ns ? __ldcg(rows + (long)sp * (D / 4)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    };
    const auto load_ml = [&](int sp, float &m, float &l) {
        m = sp < ns ? __ldcg(gm + sp) : -INFINITY;
        l = sp < ns ? __ldcg(gl + sp) : 0.0f;
    };
    float m0, l0, m1, l1, M, lsum;
    load_ml(lane, m0, l0);
    load_ml(lane + 32, m1, l1);
    load_rows(0);
    M = fmaxf(m0, m1);
#pragma unroll 1
    for (int sp = lane + 64; sp < ns; sp += 32) M = fmaxf(M, __ldcg(gm + sp));
    M = warp_max(M);
    const auto scale_of = [&](int sp, float m) {
        const float sc = m == -INFINITY ? 0.0f : fexp(m - M);
        if (sp < ns) s_sc[sp] = sc;
        return sc;
    };
    lsum = fmaf(l1, scale_of(lane + 32, m1), l0 * scale_of(lane, m0));
#pragma unroll 1
    for (int sp = lane + 64; sp < ns; sp += 32) {
        float m, l;
        load_ml(sp, m, l);
        lsum = fmaf(l, scale_of(sp, m), lsum);
    }
    lsum = warp_sum(lsum);
    if (lane == 0 && part == 0) {
        s_l[g] = lsum;
        if (ws.partial_out != nullptr && (((flagged >> g) & 1u) != 0) == dense_role) {
            const int h = head0 + g;
            if (push_c) {
                for (int p = 0; p < ws.peer_world; ++p) {
                    ws.peer_partial[p][(long)h * CQA_PARTIAL_STRIDE] = M;
                    ws.peer_partial[p][(long)h * CQA_PARTIAL_STRIDE + 1] = lsum;
                }
            } else {
                ws.partial_out[(long)h * CQA_PARTIAL_STRIDE] = M;
                ws.partial_out[(long)h * CQA_PARTIAL_STRIDE + 1] = lsum;
            }
        }
    }
    __syncwarp();
    float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 1
    for (int first = 0; first < ns; first += BATCH * nparts) {
        if (first > 0) load_rows(first);            // more splits than one batch covers
#pragma unroll
        for (int j = 0; j < BATCH; ++j) {
            const int sp = first + part + j * nparts;
            if (sp < ns) {
                const float sc = s_sc[sp];
                a.x = fmaf(buf[j].x, sc, a.x);
                a.y = fmaf(buf[j].y, sc, a.y);
                a.z = fmaf(buf[j].z, sc, a.z);
                a.w = fmaf(buf[j].w, sc, a.w);
            }
        }
    }
    reinterpret_cast<float4 *>(s_part + warp * D)[lane] = a;
    __syncthreads();
    for (int item = tid; item < nh * D; item += ATT_THREADS) {
        const int gg = item / D, ch = item % D, h = head0 + gg;
        if ((((flagged >> gg) & 1u) != 0) != dense_role) continue;
        float acc = 0.0f;
        for (int p = 0; p < nparts; ++p) acc += s_part[(gg * nparts + p) * D + ch];
        if (ws.partial_out != nullptr) {
            // un-normalised: merged across ranks later
            if (push_c) {
                for (int p = 0; p < ws.peer_world; ++p) ws.peer_partial[p][(long)h * CQA_PARTIAL_STRIDE + 2 + ch] = acc;
            } else {
                ws.partial_out[(long)h * CQA_PARTIAL_STRIDE + 2 + ch] = acc;
            }
            continue;
        }
        const float l = s_l[gg];
        ws.out[(long)h * D + ch] = acc / (l > 0.0f ? l : 1.0f);
    }
    __syncthreads();
    if (push_c && tid == 0) {
        // Exchange C: one arrival per KV head (regular merges) plus one per densely recomputed head; the last one
        // tells every rank that this rank's partial rows have landed
        __threadfence_system();
        int expected = kv_heads;
        if (ws.dense_splits > 0 && ws.cert != nullptr) expected += ws.any_flags[2] ? n_heads_total : ws.any_flags[4];
        const int t = atomicAdd(ws.peer_ticket_c, arrivals);
        if (t == expected - arrivals) {
            *ws.peer_ticket_c = 0;
            __threadfence_system();
            for (int p = 0; p < ws.peer_world; ++p)
                if (p != ws.peer_rank) st_release_sys(ws.peer_flag_c[p], ws.peer_step);
        }
    }
}

// Returns true in every thread of the CTA that took the last ticket (the bits of `mask` count them).
__device__ __forceinline__ bool take_ticket(int *ticket, int total, int *s_flag, int mask = -1)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();                  // the barrier before it orders the CTA's partials
        const int last = (atomicAdd(ticket, 1) & mask) == total - 1 ? 1 : 0;
        if (last) {
            __threadfence();
            atomicSub(ticket, total);     // ready for the next launch
        }
        *s_flag = last;
    }
    __syncthreads();
    return *s_flag != 0;
}

template <typename T2>
__device__ __forceinline__ void prefetch_rows(const T2 *blk, int lane)
{
    // a block's rows are contiguous: 128 bytes per lane and round
#pragma unroll
    for (int i = 0; i < (int)sizeof(T2) / 2; ++i)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char *>(blk) + (i * 32 + lane) * 128));
}

template <int G, typename T2>
__device__ __forceinline__ void attend_body(const cqa_cache &c, const cqa_workspace &ws, const void *q, int q_dtype, long nq,
                                            long nact, long num_tokens, int last_valid, float q_scale, int blocks_per_split)
{
    using LY = AttLayout<G, T2>;
    using Warp = AttWarp<G, T2>;
    constexpr int HG = LY::HG, SUBS = LY::SUBS;
    extern __shared__ __align__(128) char dsm[];
    __shared__ int s_flag;
    __shared__ float s_qn[4];
    const int kv = (int)blockIdx.y / SUBS, sub = (int)blockIdx.y % SUBS, head0 = kv * G + sub * HG;
    const int ns = ws.num_splits, split = (int)blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int b_begin = split * blocks_per_split;
    const int b_end = split < ns ? min((int)nact, b_begin + blocks_per_split) : b_begin;      // CTAs x >= ns: dense recompute only
    // A warp takes pairs of blocks (fewer and wider copies, half the loop overhead), single blocks where a split has so
    // few that pairs would leave warps idle (1000 tokens fp32: 47.3 -> 43.8 us a step; a line at 64 blocks measured the
    // same).
    const int unit = blocks_per_split <= ATT_WARPS ? 1 : 2, stride = unit * ATT_WARPS;
    const int my_first = b_begin + unit * warp;     // this warp's units: my_first + stride * it
    char *ring = dsm, *wring = ring + warp * ATT_STAGES * LY::STAGE;
    char *qfrag = dsm + LY::RING_BYTES;
    float *wtile = reinterpret_cast<float *>(dsm + LY::RING_BYTES + LY::QFRAG + warp * LY::WTILE);
    const unsigned wring_addr = smem_u32(wring);

    // start the pipeline before anything else
    AttIssuer<G, T2> issuer;
    issuer.init(c, ws.token_scores, (int)nq, kv, sub, my_first, b_end, unit, lane);
#pragma unroll
    for (int s = 0; s < ATT_STAGES - 1; ++s) issuer.issue(wring + s * LY::STAGE, lane);

    // the query of another group of heads (dense recompute) replaces these fragments later
    const auto load_query = [&](int h0) -> bool {
        bool third = false;
        if constexpr (LY::F32) {
            for (int i = threadIdx.x; i < HG * D; i += ATT_THREADS) reinterpret_cast<float *>(qfrag)[i] = load_q(q, q_dtype, (long)h0 * D + i);
        } else {
            if constexpr (Warp::F16) {
                // fp16 pieces: each head's query is scaled by a power of two so that its largest element is near 2^10
                if (warp < HG) {
                    float mx = 0.0f;
                    for (int i = lane; i < D; i += 32) mx = fmaxf(mx, fabsf(load_q(q, q_dtype, (long)(h0 + warp) * D + i)));
                    mx = warp_max(mx);
                    const int e = min(max((int)(__float_as_uint(mx) >> 23), 40), 220);
                    if (lane == 0) s_qn[warp] = __uint_as_float((unsigned)(254 + 10 - e) << 23);     // 2^(10 - exponent)
                }
                __syncthreads();
            }
            uint2 *frag = reinterpret_cast<uint2 *>(qfrag);
            const int step = threadIdx.x >> 5, ql = threadIdx.x & 31, hq = (ql >> 2) & 3, piece = ql >> 4;
            const int ch = 32 * (step >> 1) + 8 * (ql & 3) + 4 * (step & 1);
            float2 a = make_float2(0.0f, 0.0f), b = a;
            if (hq < HG) {
                const long o = (long)(h0 + hq) * D + ch;
                a = make_float2(load_q(q, q_dtype, o), load_q(q, q_dtype, o + 1));
                b = make_float2(load_q(q, q_dtype, o + 2), load_q(q, q_dtype, o + 3));
            }
            if constexpr (Warp::F16) {
                const float s = hq < HG ? s_qn[hq] : 0.0f;
                uint2 hi, lo;
                split_f16(__fmul2_rn(a, make_float2(s, s)), hi.x, lo.x);
                split_f16(__fmul2_rn(b, make_float2(s, s)), hi.y, lo.y);
                frag[step * 32 + ql] = piece ? lo : hi;
            } else {
                uint2 hi, mid, lo;
                split_bf16(a, hi.x, mid.x, lo.x);
                split_bf16(b, hi.y, mid.y, lo.y);
                frag[step * 32 + ql] = piece ? mid : hi;
                frag[(8 + step) * 32 + ql] = piece ? make_uint2(0u, 0u) : lo;
                third = ((lo.x | lo.y) & 0x7fff7fffu) != 0;
            }
        }
        return __syncthreads_or(third) != 0;
    };
    bool third = load_query(head0);
    // fp16: the logits of head g come out scaled like its query
    const auto unscale_logits = [&](float *sc, unsigned km) {
        if constexpr (Warp::F16) {
            for (int i = lane; i < HG * BS; i += 32)
                if (km & (1u << (i / BS))) sc[i] *= 1.0f / s_qn[i / BS];
            __syncwarp();
        }
    };

    // Softmax reference: the largest Phase-1 block maximum over the warp's blocks.  Weight scale F: the largest value
    // norm nu bounds a group's range by 2 nu, its INT4 scale by 2 nu / 15.
    const int n_my = my_first < b_end ? (b_end - my_first + stride - 1) / stride : 0;     // units
    const bool have_mb = ws.m_b != nullptr, have4 = c.values_int4_packed != nullptr;
    const long mb_ld = ws.shard_chunk > 0 ? ws.shard_chunk : ws.ld;   // a rank's own rows of the exchange buffer
    float m_init = -INFINITY, F = 32768.0f;
    {
        float mx[HG], nu = 0.0f;
#pragma unroll
        for (int g = 0; g < HG; ++g) mx[g] = -INFINITY;
        for (int b = my_first + (lane / unit) * stride + lane % unit; b < b_end && b < (int)nq; b += 32 * ATT_WARPS) {
            if (have_mb) {
#pragma unroll
                for (int g = 0; g < HG; ++g) mx[g] = fmaxf(mx[g], ws.m_b[(long)(head0 + g) * mb_ld + b]);
            }
            if (have4 && c.values_norm_max) nu = fmaxf(nu, c.values_norm_max[(long)kv * c.max_blocks + b]);
        }
#pragma unroll
        for (int g = 0; g < HG; ++g) {
            const float v = warp_max(mx[g]);
            if (g == ((lane >> 2) & 3)) m_init = v;
        }
        float bound = warp_max(nu) * 0.135f;       // 2 / 15 with room for the rounding of values and scales to fp16
        if (have4 && !c.values_norm_max) {         // caches without norms: the scales themselves
            float s = 0.0f;
            for (int i0 = 0; i0 < unit * n_my; ++i0) {
                const long b = my_first + (i0 / unit) * stride + i0 % unit;
                if (b >= b_end || b >= nq) break;
                const __half2 *row = reinterpret_cast<const __half2 *>(c.values_int4_scales + ((long)kv * c.cap_tokens + b * BS) * NG);
                for (int i = lane; i < BS * NG / 2; i += 32) { const float2 v = __half22float2(row[i]); s = fmaxf(s, fmaxf(fabsf(v.x), fabsf(v.y))); }
            }
            bound = warp_max(s);
        }
        if (have4) {
            // F * bound below 2^15
            const int e = min(max((int)(__float_as_uint(bound) >> 23) - 127, -30), 20);
            F = fminf(F, __uint_as_float((unsigned)(127 + 14 - e) << 23));
        }
    }
    Warp W;
    W.init(lane, m_init, F);

    // Everything above reads what the append and score kernels wrote (they completed before the selector, the
    // previous kernel of the chain, began); the masks and flags below are the selector's, so wait for it here.
    // CTAs that were scheduled while the selector was still running have their first blocks in flight by now.
    grid_dependency_wait();

    // Heads that are recomputed densely: their rows come from the dense pass below, nothing promoted is read for them.
    const bool dense_on = ws.dense_splits > 0 && ws.cert != nullptr;
    const bool dense_all = dense_on && ws.any_flags[2] != 0;
    const int n_dense = dense_all ? c.kv_heads * G : (dense_on ? ws.any_flags[4] : 0);
    unsigned flagged = 0;        // of the KV head's G heads; without the dense pass their rows are another call's
    if (n_dense > 0 || (ws.cert != nullptr && !dense_on)) {
        const int f = lane < G ? (ws.any_flags[2] != 0 || ws.cert[kv * G + lane].dense) : 0;
        flagged = __ballot_sync(FULL, f != 0);
    }
    const unsigned skip = dense_on ? (flagged >> (sub * HG)) & ((1u << HG) - 1u) : 0u;

    // Lane j keeps the key / value promotion bits of the warp's unit (it0 + j), one bit per head; they are re-read every
    // 32 units.
    unsigned my_masks = 0;   // km | vm << 8 of the unit's first block, the same << 16 of its second
    const auto load_masks = [&](int it0) {
        my_masks = 0;
#pragma unroll 1
        for (int i = 0; i < unit; ++i) {
            const int b = my_first + (it0 + lane) * stride + i;
            unsigned km = 0, vm = 0;
            if (b < b_end) {
#pragma unroll
                for (int g = 0; g < HG; ++g) {
                    const long o = (long)(head0 + g) * ws.ld + b;
                    km |= (ws.topk_mask[o] || b >= nq) ? (1u << g) : 0u;
                    vm |= ws.value_mask[o] ? (1u << g) : 0u;
                }
                if (b < nq) { km &= ~skip; vm &= ~skip; }
            }
            my_masks |= (km | (vm << 8)) << (16 * i);
        }
    };
    load_masks(0);
    // Tier-2 rows that will be needed are requested into L2 two units ahead (device memory only).
    const auto prefetch = [&](int it) {
        const unsigned mk = __shfl_sync(FULL, my_masks, it & 31);
        if (mk == 0) return;
        const long b = my_first + it * stride;
#pragma unroll 1
        for (int i = 0; i < unit; ++i) {
            const unsigned m = (mk >> (16 * i)) & 0xFFFFu;
            if ((m & 0xFFu) && !c.key_slots) prefetch_rows<T2>(t2_key_block<T2>(c, kv, b + i), lane);
            if ((m >> 8) && !c.value_slots) prefetch_rows<T2>(t2_value_block<T2>(c, kv, b + i), lane);
        }
    };
    for (int it = 0; it < 2 && it < n_my; ++it) prefetch(it);

#pragma unroll 1
    for (int it = 0; it < n_my; ++it) {
        const unsigned pair_masks = __shfl_sync(FULL, my_masks, it & 31);
        const int b0 = my_first + it * stride;
        char *st = wring + (it % ATT_STAGES) * LY::STAGE;
        const unsigned st_addr = wring_addr + (it % ATT_STAGES) * LY::STAGE;
        att_wait<ATT_STAGES - 2>();
        __syncwarp();    // pair `it` has landed for every lane, and every lane is done with the slot refilled next
        issuer.issue(wring + ((it + ATT_STAGES - 1) % ATT_STAGES) * LY::STAGE, lane);
        if (((it + 2) & 31) > 1 && it + 2 < n_my) prefetch(it + 2);      // within the 32 pairs whose masks are at hand
#pragma unroll 1
        for (int i = 0; i < unit; ++i) {
            const int b = b0 + i;
            if (b >= b_end) break;
            const unsigned km = (pair_masks >> (16 * i)) & 0xFFu, vm = (pair_masks >> (16 * i + 8)) & 0xFFu;
            const int n_valid = (b == (int)nact - 1) ? last_valid : BS;
            float *sc = reinterpret_cast<float *>(st + LY::SCORES + i * LY::SCORES_BLK);
            if (km) {
                W.key_logits(t2_key_block<T2>(c, kv, b), km, n_valid, q_scale, qfrag, third, sc);
                unscale_logits(sc, km);
            }
            float2 w0, w1;
            W.weights(sc, km != 0 || !have_mb, w0, w1);
            if (have4 && b < (int)nq && vm != (1u << HG) - 1u)
                W.int4_values(st_addr + LY::PACKED + i * LY::PACKED_BLK, st + LY::SCALES + i * LY::SCALES_BLK,
                              st_addr + LY::SCALES + i * LY::SCALES_BLK, st_addr + LY::ZEROS + i * LY::SCALES_BLK,
                              ((vm >> W.h) & 1u) ? 0.0f : 1.0f, w0, w1);
            if (vm) W.t2_values(t2_value_block<T2>(c, kv, b), vm, n_valid, w0, w1, wtile);
        }
        if ((it & 31) == 31 && it + 1 < n_my) {
            load_masks(it + 1);
            for (int i = 1; i <= 2 && it + i < n_my; ++i) prefetch(it + i);
        }
    }
    att_wait<0>();
    float *sm_m = reinterpret_cast<float *>(ring);
    float *sm_l = sm_m + ATT_WARPS * HG;
    float *sm_acc = sm_l + ATT_WARPS * HG;
    if (split < ns) {
        __syncthreads();  // the ring is reused as merge buffers
        W.store(sm_m, sm_l, sm_acc, warp);
        cta_merge_store<HG>(sm_m, sm_l, sm_acc, ws.part_m, ws.part_l, ws.part_acc, head0, split, ns);
        if (take_ticket(ws.tickets + kv, ns * SUBS, &s_flag))
            final_merge(ws.part_m, ws.part_l, ws.part_acc, ns, kv * G, G, ws, false, flagged, reinterpret_cast<float *>(ring), c.kv_heads,
                        c.kv_heads * G);
    }
    if (n_dense == 0) return;

    // ---- dense recompute of the flagged heads: units of (group of heads with a flagged one, chunk of blocks); the heads
    // of a group share the rows.  A CTA draws its next unit from a counter when it is done with the last one (the splits
    // end far apart where their promotions differ, and the CTAs that merge come later still; dealt out by CTA number a step
    // of 8192 tokens fp32 took 69.7 us in place of 64.2, four sequences of 65536 tokens 402 in place of 375).  The counter is the upper 24 bits of the first group's ticket
    // word: each CTA draws one number past the last unit, and the one with the largest sets it back.
    constexpr int WINDOW = 256;          // groups looked at together
    __shared__ unsigned char s_group[WINDOW], s_heads[WINDOW];
    __shared__ int s_count, s_unit;
    const int groups = c.kv_heads * SUBS, ds = ws.dense_splits;
    const int n_ctas = (int)gridDim.x * groups;
    int *counter = ws.tickets + c.kv_heads;
    constexpr int UNIT_SHIFT = 8;
    static_assert(CQA_MAX_DENSE_SPLITS < (1 << UNIT_SHIFT), "the ticket is the lower bits of the word");
    const auto draw = [&] { if (threadIdx.x == 0) s_unit = (int)((unsigned)atomicAdd(counter, 1 << UNIT_SHIFT) >> UNIT_SHIFT); };
    draw();
    int units_before = 0;
    const long nblk = (num_tokens + BS - 1) / BS, bps = (nblk + ds - 1) / ds;
    int loaded = (int)blockIdx.y;
#pragma unroll 1
    for (int g0 = 0; g0 < groups; g0 += WINDOW) {
        const int in_window = min(groups - g0, WINDOW);
        __syncthreads();
        if ((int)threadIdx.x < in_window) {
            unsigned heads = 0;
            const int y = g0 + (int)threadIdx.x, dh0 = (y / SUBS) * G + (y % SUBS) * HG;
#pragma unroll
            for (int g = 0; g < HG; ++g) heads |= (dense_all || ws.cert[dh0 + g].dense) ? 1u << g : 0u;
            s_heads[threadIdx.x] = (unsigned char)heads;
        }
        __syncthreads();
        if (warp == 0) {
            int n = 0;
            for (int i = 0; i < in_window; i += 32) {
                const bool f = i + lane < in_window && s_heads[i + lane] != 0;
                const unsigned who = __ballot_sync(FULL, f);
                if (f) s_group[n + __popc(who & ((1u << lane) - 1u))] = (unsigned char)(i + lane);
                n += __popc(who);
            }
            if (lane == 0) s_count = n;
        }
        __syncthreads();
        const int n_groups = s_count;
#pragma unroll 1
        for (;;) {
            const int u = s_unit - units_before;
            if (u >= n_groups * ds) break;
            const int at = s_group[u % n_groups], chunk = u / n_groups, y = g0 + at;
            const unsigned heads = s_heads[at];
            const int dkv = y / SUBS, dh0 = dkv * G + (y % SUBS) * HG;
            if (loaded != y) {
                __syncthreads();
                third = load_query(dh0);
                loaded = y;
            }
            const long d0 = (long)chunk * bps, d1 = min(nblk, d0 + bps);
            W.init(lane, -INFINITY, 32768.0f);
            float *sc = reinterpret_cast<float *>(wring + LY::SCORES);
            for (int i = lane; i < 4 * BS; i += 32) sc[i] = 0.0f;
            __syncwarp();
#pragma unroll 1
            for (long b = d0 + warp; b < d1; b += ATT_WARPS) {
                const T2 *kblk = t2_key_block<T2>(c, dkv, b), *vblk = t2_value_block<T2>(c, dkv, b);
                if (kblk == nullptr || vblk == nullptr) continue;
                if (!c.value_slots) prefetch_rows<T2>(vblk, lane);
                if (b + ATT_WARPS < d1 && !c.key_slots) prefetch_rows<T2>(t2_key_block<T2>(c, dkv, b + ATT_WARPS), lane);
                const int n_valid = (int)min((long)BS, num_tokens - b * BS);
                W.key_logits(kblk, heads, n_valid, q_scale, qfrag, third, sc);
                unscale_logits(sc, heads);
                float2 w0, w1;
                W.weights(sc, true, w0, w1);
                W.t2_values(vblk, heads, n_valid, w0, w1, wtile);
                __syncwarp();
            }
            __syncthreads();
            draw();
            W.store(sm_m, sm_l, sm_acc, warp);
            cta_merge_store<HG>(sm_m, sm_l, sm_acc, ws.dense_m, ws.dense_l, ws.dense_acc, dh0, chunk, ds);
            if (take_ticket(ws.tickets + c.kv_heads + dh0, ds, &s_flag, (1 << UNIT_SHIFT) - 1))
                final_merge(ws.dense_m, ws.dense_l, ws.dense_acc, ds, dh0, HG, ws, true, heads, reinterpret_cast<float *>(ring), c.kv_heads,
                            c.kv_heads * G, __popc(heads));
            __syncthreads();      // the ring is merge scratch
        }
        units_before += n_groups * ds;
    }
    if (threadIdx.x == 0 && s_unit == units_before + n_ctas - 1) atomicSub(counter, (units_before + n_ctas) << UNIT_SHIFT);
}

template <int G, typename T2>
__global__ void __launch_bounds__(ATT_THREADS, CQA_ATT_MIN_CTAS) attend_kernel(cqa_cache c, cqa_workspace ws, const void *q,
                                                               int q_dtype, long nq, long nact, long num_tokens,
                                                               int last_valid, float q_scale, int blocks_per_split)
{
    attend_body<G, T2>(c, ws, q, q_dtype, nq, nact, num_tokens, last_valid, q_scale, blocks_per_split);
}

// Sequence blockIdx.z of a batch.  grid.x = the largest split count of the batch; CTAs beyond a
// sequence's own split count have nothing to do.
template <int G, typename T2>
__global__ void __launch_bounds__(ATT_THREADS, CQA_ATT_MIN_CTAS) attend_batched_kernel(const cqa_batch_item *items, int q_dtype,
                                                                                      float q_scale, int do_append)
{
    const cqa_batch_item &it = *stage_batch_item(items + blockIdx.z);
    const long num_tokens = it.pos + do_append;
    const long nq = num_tokens / BS, nact = (num_tokens + BS - 1) / BS;
    const int ns = it.ws.num_splits;
    const int last_valid = nact == nq ? BS : (int)(num_tokens - nq * BS);
    attend_body<G, T2>(it.cache, it.ws, it.q, q_dtype, nq, nact, num_tokens, last_valid, q_scale, (int)((nact + ns - 1) / ns));
}

// Columns of CTAs beside the splits that only take part in the dense recompute: what fits the first wave, at most
// eight.  A short context leaves most of the GPU idle, and a recompute behind the splits of a few CTAs cost it 8 us;
// a long one fills the GPU with splits, and the recompute follows on all of them.
static int spare_columns(int splits, long rows)
{
    const long slots = (long)sm_count() * CQA_ATT_MIN_CTAS, left = slots - rows * splits;
    return (int)(left <= 0 ? 0 : (left / rows < 8 ? left / rows : 8));
}

template <int G, typename T2>
static size_t attend_smem() { return ((size_t)AttLayout<G, T2>::TOTAL + 15) & ~(size_t)15; }

template <int G, typename T2>
static int attend_launch_gt(const cqa_cache *c, const cqa_workspace *ws, const void *q, int q_dtype, long nq,
                            long nact, long num_tokens, int last_valid, float q_scale, cudaStream_t st, bool chained)
{
    const int ns = ws->num_splits;
    const int bps = (int)((nact + ns - 1) / ns);
    const bool dense = ws->cert && ws->dense_splits > 0 && ws->dense_m && ws->dense_l && ws->dense_acc;
    cqa_workspace w = *ws;
    if (!dense) w.dense_splits = 0;
    const size_t smem = attend_smem<G, T2>();
    static size_t granted[SMEM_ATTR_DEVICES] = {};
    const int rc_attr = check_cuda(ensure_dynamic_smem(attend_kernel<G, T2>, smem, granted), "cudaFuncSetAttribute(attend_kernel)");
    if (rc_attr) return rc_attr;
    const int rows = c->kv_heads * AttLayout<G, T2>::SUBS;
    dim3 grid((unsigned)(ns + (dense ? spare_columns(ns, rows) : 0)), (unsigned)rows);
    return check_cuda(launch_chained(attend_kernel<G, T2>, grid, dim3(ATT_THREADS), smem, st, chained, *c, w, q, q_dtype, nq,
                                     nact, num_tokens, last_valid, q_scale, bps),
                      "attend_kernel");
}

template <typename T2>
static int attend_launch_t(const cqa_cache *c, const cqa_workspace *ws, const void *q, int q_dtype, long nq,
                           long nact, long num_tokens, int last_valid, float q_scale, cudaStream_t st, bool chained)
{
    switch (c->gqa_group) {
    case 1: return attend_launch_gt<1, T2>(c, ws, q, q_dtype, nq, nact, num_tokens, last_valid, q_scale, st, chained);
    case 2: return attend_launch_gt<2, T2>(c, ws, q, q_dtype, nq, nact, num_tokens, last_valid, q_scale, st, chained);
    case 4: return attend_launch_gt<4, T2>(c, ws, q, q_dtype, nq, nact, num_tokens, last_valid, q_scale, st, chained);
    case 8: return attend_launch_gt<8, T2>(c, ws, q, q_dtype, nq, nact, num_tokens, last_valid, q_scale, st, chained);
    }
    set_error("cqa_attend: unsupported gqa_group %d", c->gqa_group);
    return CQA_ERR_UNSUPPORTED;
}

// Argument checks of Phase 2 (also called by the fused step before its first launch).
int attend_check(const cqa_cache *c, const cqa_workspace *ws, long nq, long nact, int last_valid)
{
    if (ws->num_splits <= 0 || !ws->part_m || !ws->part_l || !ws->part_acc || (!ws->out && !ws->partial_out) || !ws->topk_mask ||
        !ws->value_mask || !ws->tickets) {
        set_error("cqa_attend: workspace is missing partial buffers, tickets, masks or the output");
        return CQA_ERR_INVALID;
    }
    if (nq > 0 && !ws->token_scores) { set_error("cqa_attend: token_scores missing"); return CQA_ERR_INVALID; }
    if (((uintptr_t)ws->token_scores | (uintptr_t)c->values_int4_packed | (uintptr_t)c->values_int4_scales |
         (uintptr_t)c->values_int4_zeros) & 15) {
        set_error("cqa_attend: token_scores and the INT4 value arrays must be 16-byte aligned (16-byte copies)");
        return CQA_ERR_INVALID;
    }
    if (nq < 0 || nact <= 0 || nact < nq || nact > ws->ld || nact > c->max_blocks) {
        set_error("cqa_attend: nact=%ld out of range (nq=%ld, ld=%ld, max_blocks=%ld)", nact, nq, (long)ws->ld,
                  (long)c->max_blocks);
        return CQA_ERR_INVALID;
    }
    if (ws->num_splits > CQA_MAX_SPLITS || ws->dense_splits > CQA_MAX_DENSE_SPLITS) {
        set_error("cqa_attend: at most %d splits and %d dense splits", CQA_MAX_SPLITS, CQA_MAX_DENSE_SPLITS);
        return CQA_ERR_TOO_LARGE;
    }
    if (ws->num_splits > nact) { set_error("cqa_attend: more splits (%d) than blocks (%ld)", ws->num_splits, nact); return CQA_ERR_INVALID; }
    if (last_valid < 1 || last_valid > BS) { set_error("cqa_attend: last_block_valid=%d", last_valid); return CQA_ERR_INVALID; }
    if (!c->keys_t2 || !c->values_t2) {
        set_error("cqa_attend: Tier-2 key/value arrays are required (promoted and trailing blocks read them)");
        return CQA_ERR_INVALID;
    }
    // A certificate can flag heads for the dense recompute; their rows are then written by the dense recompute only.
    // Without the dense scratch nothing would write them, so that combination is refused instead of leaving
    // stale rows in the output.
    if (ws->cert != nullptr && (ws->dense_splits <= 0 || !ws->dense_m || !ws->dense_l || !ws->dense_acc)) {
        set_error("cqa_attend: a certificate is attached (ws->cert) but the dense-recompute scratch "
                  "(dense_splits, dense_m, dense_l, dense_acc) is missing; pass it, or detach the certificate");
        return CQA_ERR_INVALID;
    }
    if (ws->cert != nullptr && !ws->any_flags) { set_error("cqa_attend: certificate without flag words"); return CQA_ERR_INVALID; }
    if (c->t2_dtype < 0 || c->t2_dtype > 2) { set_error("cqa_attend: unknown Tier-2 dtype %d", c->t2_dtype); return CQA_ERR_INVALID; }
    return CQA_OK;
}

// `chained`: the previous kernel on the stream is the selector of the same fused step, so the kernel may be
// scheduled early and stage its first blocks (written two kernels back) before waiting for the selector.
int attend_launch(const cqa_cache *c, const cqa_workspace *ws, const void *q, int q_dtype, long nq, long nact,
                  long num_tokens, int last_valid, float q_scale, cudaStream_t st, bool chained)
{
    const int rc = attend_check(c, ws, nq, nact, last_valid);
    if (rc) return rc;
    switch (c->t2_dtype) {
    case CQA_F32: return attend_launch_t<float>(c, ws, q, q_dtype, nq, nact, num_tokens, last_valid, q_scale, st, chained);
    case CQA_F16: return attend_launch_t<__half>(c, ws, q, q_dtype, nq, nact, num_tokens, last_valid, q_scale, st, chained);
    default: return attend_launch_t<__nv_bfloat16>(c, ws, q, q_dtype, nq, nact, num_tokens, last_valid, q_scale, st, chained);
    }
}

template <int G, typename T2>
static int attend_batched_launch_gt(const cqa_batch_item *items_dev, int n_items, int kv_heads, int max_splits, int q_dtype,
                                    float q_scale, int do_append, cudaStream_t st)
{
    const size_t smem = attend_smem<G, T2>();
    static size_t granted[SMEM_ATTR_DEVICES] = {};
    const int rc = check_cuda(ensure_dynamic_smem(attend_batched_kernel<G, T2>, smem, granted),
                              "cudaFuncSetAttribute(attend_batched_kernel)");
    if (rc) return rc;
    const int rows = kv_heads * AttLayout<G, T2>::SUBS;
    dim3 grid((unsigned)(max_splits + spare_columns(max_splits, (long)rows * n_items)), (unsigned)rows, (unsigned)n_items);
    return check_cuda(launch_chained(attend_batched_kernel<G, T2>, grid, dim3(ATT_THREADS), smem, st, true, items_dev, q_dtype,
                                     q_scale, do_append), "attend_batched_kernel");
}

template <typename T2>
static int attend_batched_launch_t(const cqa_batch_item *items_dev, int n_items, int kv_heads, int gqa_group, int max_splits,
                                   int q_dtype, float q_scale, int do_append, cudaStream_t st)
{
    switch (gqa_group) {
    case 1: return attend_batched_launch_gt<1, T2>(items_dev, n_items, kv_heads, max_splits, q_dtype, q_scale, do_append, st);
    case 2: return attend_batched_launch_gt<2, T2>(items_dev, n_items, kv_heads, max_splits, q_dtype, q_scale, do_append, st);
    case 4: return attend_batched_launch_gt<4, T2>(items_dev, n_items, kv_heads, max_splits, q_dtype, q_scale, do_append, st);
    case 8: return attend_batched_launch_gt<8, T2>(items_dev, n_items, kv_heads, max_splits, q_dtype, q_scale, do_append, st);
    }
    set_error("cqa_layer_step_batched: unsupported gqa_group %d", gqa_group);
    return CQA_ERR_UNSUPPORTED;
}

// Phase 2 of a batch; every item was checked by the caller (attend_check) and carries the dense scratch.
int attend_batched_launch(const cqa_batch_item *items_dev, int n_items, int kv_heads, int gqa_group, int t2_dtype,
                          int max_splits, int q_dtype, float q_scale, int do_append, cudaStream_t st)
{
    switch (t2_dtype) {
    case CQA_F32: return attend_batched_launch_t<float>(items_dev, n_items, kv_heads, gqa_group, max_splits, q_dtype, q_scale, do_append, st);
    case CQA_F16: return attend_batched_launch_t<__half>(items_dev, n_items, kv_heads, gqa_group, max_splits, q_dtype, q_scale, do_append, st);
    default: return attend_batched_launch_t<__nv_bfloat16>(items_dev, n_items, kv_heads, gqa_group, max_splits, q_dtype, q_scale, do_append, st);
    }
}

// Dense recompute alone (no splits), for the heads the attached
// certificate lists (cert[h].dense with the list in any_flags[5..], or every head when any_flags[2] is set).
template <typename T2>
static int dense_launch_t(const cqa_cache *c, const cqa_workspace *ws, const void *q, int q_dtype, long num_tokens,
                          float q_scale, cudaStream_t st)
{
    cqa_workspace w = *ws;
    w.num_splits = 0;
    const long nblk = (num_tokens + BS - 1) / BS;
#define CQA_DENSE_CASE(GG)                                                                                             \
    case GG: {                                                                                                         \
        const int rows = c->kv_heads * AttLayout<GG, T2>::SUBS;                                                        \
        dim3 grid((unsigned)((sm_count() * CQA_ATT_MIN_CTAS + rows - 1) / rows), (unsigned)rows);                      \
        const size_t smem = attend_smem<GG, T2>();                                                                         \
        static size_t granted[SMEM_ATTR_DEVICES] = {};                                                                 \
        const int rc = check_cuda(ensure_dynamic_smem(attend_kernel<GG, T2>, smem, granted), "cudaFuncSetAttribute(attend_kernel)"); \
        if (rc) return rc;                                                                                             \
        return check_cuda(launch_chained(attend_kernel<GG, T2>, grid, dim3(ATT_THREADS), smem, st, false, *c, w, q, q_dtype, \
                                         (long)0, nblk, num_tokens, BS, q_scale, 1), "attend_kernel (dense)");         \
    }
    switch (c->gqa_group) {
        CQA_DENSE_CASE(1)
        CQA_DENSE_CASE(2)
        CQA_DENSE_CASE(4)
        CQA_DENSE_CASE(8)
    }
#undef CQA_DENSE_CASE
    set_error("cqa_dense_attend: unsupported gqa_group %d", c->gqa_group);
    return CQA_ERR_UNSUPPORTED;
}

int dense_launch(const cqa_cache *c, const cqa_workspace *ws, const void *q, int q_dtype, long num_tokens, float q_scale,
                 cudaStream_t st)
{
    if (!ws->cert || !ws->any_flags || ws->dense_splits <= 0 || ws->dense_splits > CQA_MAX_DENSE_SPLITS || !ws->dense_m ||
        !ws->dense_l || !ws->dense_acc || !ws->tickets || !ws->out) {
        set_error("cqa_dense_attend: needs cert, any_flags, the dense scratch (1..%d splits), tickets and out",
                  CQA_MAX_DENSE_SPLITS);
        return CQA_ERR_INVALID;
    }
    const bool identity = c->key_slots == nullptr && c->value_slots == nullptr;
    if (num_tokens <= 0 || (num_tokens + BS - 1) / BS > c->max_blocks ||
        (identity && (num_tokens > c->keys_t2_rows || num_tokens > c->values_t2_rows))) {
        set_error("cqa_dense_attend: num_tokens=%ld out of range", num_tokens);
        return CQA_ERR_INVALID;
    }
    if (!c->keys_t2 || !c->values_t2) { set_error("cqa_dense_attend: Tier-2 arrays missing"); return CQA_ERR_INVALID; }
    if (q_dtype < 0 || q_dtype > 2) { set_error("cqa_dense_attend: unknown q dtype"); return CQA_ERR_INVALID; }
    switch (c->t2_dtype) {
    case CQA_F32: return dense_launch_t<float>(c, ws, q, q_dtype, num_tokens, q_scale, st);
    case CQA_F16: return dense_launch_t<__half>(c, ws, q, q_dtype, num_tokens, q_scale, st);
    case CQA_BF16: return dense_launch_t<__nv_bfloat16>(c, ws, q, q_dtype, num_tokens, q_scale, st);
    }
    set_error("cqa_dense_attend: unknown Tier-2 dtype %d", c->t2_dtype);
    return CQA_ERR_INVALID;
}

// Merge of per-rank partial rows (max, sum, acc[128]) of every head: one CTA per head, one thread per channel.
__global__ void __launch_bounds__(D) merge_partials_kernel(const float *parts, int n_parts, int n_heads, float *out)
{
    const int h = blockIdx.x, ch = threadIdx.x;
    float M = -INFINITY;
    for (int p = 0; p < n_parts; ++p) M = fmaxf(M, parts[((long)p * n_heads + h) * CQA_PARTIAL_STRIDE]);
    float l = 0.0f, a = 0.0f;
    for (int p = 0; p < n_parts; ++p) {
        const float *row = parts + ((long)p * n_heads + h) * CQA_PARTIAL_STRIDE;
        const float sc = row[0] == -INFINITY ? 0.0f : fexp(row[0] - M);
        l = fmaf(row[1], sc, l);
        a = fmaf(row[2 + ch], sc, a);
    }
    out[(long)h * D + ch] = a / (l > 0.0f ? l : 1.0f);
}

int merge_partials_launch(const float *parts, int n_parts, int n_heads, float *out, cudaStream_t st)
{
    merge_partials_kernel<<<n_heads, D, 0, st>>>(parts, n_parts, n_heads, out); note_launch();
    return check_launch("merge_partials_kernel");
}

// ---------------------------------------------------------------------------
// Built-in scratch for cqa_attend_static: split partials and merge tickets for
// callers that cannot allocate device memory.
// Layout: [Phase-2 m | l | acc][dense m | l | acc][tickets (int32)].
constexpr long STATIC_P2 = (long)CQA_STATIC_MAX_HEADS * CQA_STATIC_MAX_SPLITS;
constexpr long STATIC_DN = (long)CQA_STATIC_MAX_HEADS * CQA_STATIC_MAX_DENSE_SPLITS;
constexpr long STATIC_TICKETS = 2 * CQA_STATIC_MAX_HEADS;
constexpr long STATIC_FLOATS = STATIC_P2 * (D + 2) + STATIC_DN * (D + 2) + STATIC_TICKETS;
static __device__ __align__(256) float g_static_partials[STATIC_FLOATS];

// Device address of g_static_partials per device.  In host code the symbol is
// only a handle; the address a kernel can use comes from cudaGetSymbolAddress,
// looked up once per device with that device current.
static float *static_partials_for_current_device(int *rc_out)
{
    constexpr int MAX_DEV = 64;
    static float *addr[MAX_DEV] = {nullptr};
    static std::mutex mu;
    int dev = -1;
    *rc_out = check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
    if (*rc_out) return nullptr;
    if (dev < 0 || dev >= MAX_DEV) {
        set_error("cqa_attend_static: device index %d out of range", dev);
        *rc_out = CQA_ERR_UNSUPPORTED;
        return nullptr;
    }
    std::lock_guard<std::mutex> lock(mu);
    if (!addr[dev]) {
        void *p = nullptr;
        *rc_out = check_cuda(cudaGetSymbolAddress(&p, g_static_partials), "cudaGetSymbolAddress(g_static_partials)");
        if (*rc_out) return nullptr;
        addr[dev] = static_cast<float *>(p);
    }
    return addr[dev];
}

int attend_static_launch(const cqa_cache *c, const cqa_workspace *ws, const void *q, int q_dtype, long nq, long nact,
                         long num_tokens, int last_valid, float q_scale, cudaStream_t st)
{
    const long H = (long)c->kv_heads * c->gqa_group;
    if (H > CQA_STATIC_MAX_HEADS || ws->num_splits > CQA_STATIC_MAX_SPLITS ||
        ws->dense_splits > CQA_STATIC_MAX_DENSE_SPLITS) {
        set_error("cqa_attend_static: %ld heads / %d splits / %d dense splits exceed the built-in scratch "
                  "(limits %d / %d / %d); use cqa_attend with caller-provided partial buffers",
                  H, ws->num_splits, ws->dense_splits, CQA_STATIC_MAX_HEADS, CQA_STATIC_MAX_SPLITS,
                  CQA_STATIC_MAX_DENSE_SPLITS);
        return CQA_ERR_TOO_LARGE;
    }
    int rc = CQA_OK;
    float *base = static_partials_for_current_device(&rc);
    if (rc) return rc;
    cqa_workspace w = *ws;
    w.part_m = base;
    w.part_l = base + STATIC_P2;
    w.part_acc = base + 2 * STATIC_P2;
    float *dn = base + STATIC_P2 * (D + 2);
    w.dense_m = dn;
    w.dense_l = dn + STATIC_DN;
    w.dense_acc = dn + 2 * STATIC_DN;
    w.tickets = reinterpret_cast<int32_t *>(dn + STATIC_DN * (D + 2));
    // The merge tickets are the only part of the shared array that must start at zero.
    rc = check_cuda(cudaMemsetAsync(w.tickets, 0, STATIC_TICKETS * sizeof(int32_t), st), "cudaMemsetAsync(tickets)");
    if (rc) return rc;
    return attend_launch(c, &w, q, q_dtype, nq, nact, num_tokens, last_valid, q_scale, st, false);
}

}  // namespace cqa
