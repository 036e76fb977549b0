// Selector and certifier: one CTA of 256, 512 or 1024 threads (NT) per (query head, role); selcert_threads has the rule.
//
// A thread owns the blocks b = tid, tid + NT, ...  The per-block values live in shared-memory arrays and every phase is
// a short rolled loop over them with one CTA barrier: the executed code is small on purpose, because ~100 CTAs start the
// same code at the same moment and an unrolled form of these loops was bound by instruction fetch.  Bound: the latency
// of the chain of phases (one sequence: 22 K cycles at 2048 blocks, 40 K at 8192) or, in a batch, issue.
//
//   role 0 (select) : exploration bits (drawn before the wait on the score
//            kernel), block masses and mass fractions (canonical sum), the 256
//            heaviest blocks (ties -> lower block id) by a radix search on the
//            float bit patterns, ordered by counting and searching; sequential
//            cumulative mass by one thread while the others write the masks without
//            a selection; K* with the Rung-1 expansion; the selected blocks' mask.
//   role 1 (ranking): query row and Delta (before the wait), top-4 blocks by
//            m_b (per-thread lists merged by shuffles), FP16 re-score of each
//            candidate by a quarter of the warps while the boundary maximum is taken,
//            ranking / boundary / score-consistency flags, work list of the
//            dense recompute.
//   role 2 (values) : Rung-2 value check: the promoted blocks are those whose
//            contribution mass*eta is at or above a threshold found by a search
//            over "column sums" (histogram hints, then two bits per step), no sort
//            and no serial walk.
//
// cqa_select, cqa_certify and the fused cqa_layer_step all launch the same
// kernel with a phase mask.  Sums over blocks use the canonical orders
// documented at the functions; prefix sums over the sorted order are
// sequential.
#include "common.cuh"
#include "rescore.cuh"

namespace cqa {

constexpr int CAND = 256;          // candidates kept by the top search
constexpr int LIST = 384;          // entries it orders at most
constexpr int HIST = 2048;         // histogram bins
constexpr int PH_SELECT = 1, PH_CERTIFY = 2;
// Sequence-sharded runs split the ranking check around an exchange: PH_TOP_ONLY stops role 1 once the top
// list is in the certificate; PH_GIVEN resumes it from that list with FP16 scores computed by the ranks that
// own the blocks (ws.given_fp16) and runs role 1 alone.
constexpr int PH_TOP_ONLY = 4, PH_GIVEN = 8;
constexpr int PH_FLAGS_CLEARED = 16;   // the caller already zeroed ws.any_flags on this stream
constexpr int PH_PEER_B = 64;          // role 1 exchanges the FP16 re-scores with the other ranks itself (ws.peer_*)

typedef unsigned long long u64;

// Philox4x32-10 on the counter (c0, head, offset) under `seed`: four 32-bit words.
__device__ __forceinline__ uint4 philox4(unsigned long long seed, unsigned long long offset, unsigned head, unsigned c0)
{
    unsigned c1 = head, c2 = (unsigned)offset, c3 = (unsigned)(offset >> 32);
    unsigned k0 = (unsigned)seed, k1 = (unsigned)(seed >> 32);
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const unsigned hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
        const unsigned hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
        const unsigned n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
        c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
    return make_uint4(c0, c1, c2, c3);
}
// The exploration draw takes one 16-bit uniform per (block, head, call): the eight blocks a thread owns in a row
// (b, b + 1024, ..., b + 7168) share one Philox call with counter word (b mod 1024) + 1024 * (b div 8192); block
// number i of the eight reads half (i mod 2) of output word i div 2.

__device__ __forceinline__ void cp_async4(float *smem, const float *gmem)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(gmem) : "memory");
}

struct SCShared {
    float red_f[2][32];
    float red_f3[2][3][32];
    unsigned red_u[2][2][32];
    int red_i[2][32];
    int bcast_i[8];
    int counter, counter2;
};

__device__ __forceinline__ u64 make_key(float v, int idx)
{
    // v >= 0: the bit pattern orders like the value; ties -> lower index first.
    return ((u64)__float_as_uint(v) << 32) | (u64)(0xFFFFFFFFu - (unsigned)idx);
}
__device__ __forceinline__ int key_idx(u64 k) { return (int)(0xFFFFFFFFu - (unsigned)(k & 0xFFFFFFFFull)); }
__device__ __forceinline__ float key_val(u64 k) { return __uint_as_float((unsigned)(k >> 32)); }
__device__ __forceinline__ unsigned orderable(float v)
{
    unsigned u = __float_as_uint(v);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ u64 shfl_xor_u64(u64 v, int m)
{
    unsigned lo = (unsigned)v, hi = (unsigned)(v >> 32);
    lo = __shfl_xor_sync(FULL, lo, m);
    hi = __shfl_xor_sync(FULL, hi, m);
    return ((u64)hi << 32) | lo;
}

// Maximum of one value per thread over the CTA, in every thread; one barrier (rows alternate with `parity`).
template <int NT>
__device__ __forceinline__ float cta_max(float v, SCShared &sh, int &parity)
{
    const unsigned u = __reduce_max_sync(FULL, orderable(v));
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) sh.red_u[parity][0][w] = u;
    __syncthreads();
    const unsigned r = __reduce_max_sync(FULL, sh.red_u[parity][0][l & (NT / 32 - 1)]);
    parity ^= 1;
    return __uint_as_float((r & 0x80000000u) ? r & 0x7FFFFFFFu : ~r);
}

// Every per-block loop of this kernel is a ROLLED loop over shared-memory arrays ("for k < nk: b = k * NT + tid").
// The code of a phase is then a few dozen instructions that stay in the instruction cache, instead of the same
// instructions unrolled once per block a thread owns: with ~100 CTAs starting the same straight-line code at the same
// moment, fetching instructions through the L2 was what bounded the unrolled form.

// Canonical sum of vals[0..n) (shared memory): 32 consecutive values by a warp butterfly (16..1), 8 such sums by a
// butterfly (4,2,1) = one leaf of 256 values, leaves added left to right.  Result in every thread.  gsum needs
// n_pad / 32 floats, leaf n_pad / 256 + 8.
template <int NT>
__device__ __forceinline__ float cta_canonical_sum(const float *vals, int n, int nk, float *gsum, float *leaf)
{
    const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
    const int ngroups = (n + 31) >> 5, nleaf = (n + 255) >> 8, nleaf8 = (nleaf + 7) & ~7;
#pragma unroll 1
    for (int k = 0; k < nk; ++k) {
        const int b = k * NT + tid;
        const float s = warp_sum(b < n ? vals[b] : 0.0f);
        if (l == 0 && k * (NT / 32) + w < ngroups) gsum[k * (NT / 32) + w] = s;   // groups beyond n hold nothing
    }
    __syncthreads();
    if (tid < nleaf8) {
        float p[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) p[i] = (tid * 8 + i) < ngroups ? gsum[tid * 8 + i] : 0.0f;
#pragma unroll
        for (int s = 4; s >= 1; s >>= 1)
#pragma unroll
            for (int i = 0; i < s; ++i) p[i] = __fadd_rn(p[i], p[i + s]);
        leaf[tid] = p[0];
    }
    __syncthreads();
    // leaves beyond the last are zero, and adding zero changes nothing; eight are fetched at a time
    float total = 0.0f;
#pragma unroll 1
    for (int L = 0; L < nleaf8; L += 8) {
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = leaf[L + i];
#pragma unroll
        for (int i = 0; i < 8; ++i) total = L + i == 0 ? v[0] : __fadd_rn(total, v[i]);
    }
    return total;
}

// In-place descending bitonic sort of n_pad (power of two) 64-bit keys by the whole CTA.
template <int NT>
__device__ __noinline__ void bitonic_sort_desc(u64 *keys, int n_pad)
{
    for (int k = 2; k <= n_pad; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = threadIdx.x; i < n_pad; i += NT) {
                const int ixj = i ^ j;
                if (ixj > i) {
                    const bool desc = (i & k) == 0;
                    const u64 a = keys[i], b = keys[ixj];
                    if (desc ? (a < b) : (a > b)) {
                        keys[i] = b;
                        keys[ixj] = a;
                    }
                }
            }
            __syncthreads();
        }
    }
}

// Orders the m <= LIST values lv[0..m) (bit patterns of floats >= 0; lv is zero up to the next multiple of 32): the place
// of entry i is the number of entries that are larger, or equal and earlier in the list (the lists are in block order,
// so ties go to the lower block id).  A warp orders 32 entries among themselves by counting; the places among the other
// groups of 32 are binary searches in their ordered values, shared by the warps that are left over.  The first CAND
// places go to cum[] (values) and sid[] (ids[i], or i without ids).  rank: LIST zeroed words, sorted: LIST words.
// (Counting over the whole list took 5.6 K cycles with 1024 threads and 13 K with 256, a bitonic network on 64-bit keys
// 5.8 K and 8 K.)
template <int NT>
__device__ __forceinline__ void order_list(const unsigned *lv, const unsigned *ids, int m, int *rank, int *sorted, float *cum, int *sid)
{
    constexpr int NW = NT / 32;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int groups = (m + 31) >> 5;
#pragma unroll 1
    for (int g = w; g < groups; g += NW) {
        const int x = (int)lv[g * 32 + lane];
        int r = 0;
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
            const int4 v = *reinterpret_cast<const int4 *>(lv + g * 32 + j);
            r += (v.x > x || (v.x == x && j < lane)) ? 1 : 0;
            r += (v.y > x || (v.y == x && j + 1 < lane)) ? 1 : 0;
            r += (v.z > x || (v.z == x && j + 2 < lane)) ? 1 : 0;
            r += (v.w > x || (v.w == x && j + 3 < lane)) ? 1 : 0;
        }
        sorted[g * 32 + r] = x;
        atomicAdd(rank + g * 32 + lane, r);
    }
    __syncthreads();
    const int parts = groups < NW ? NW / groups : 1;       // warps per group of entries
#pragma unroll 1
    for (int item = w; item < groups * parts; item += NW) {
        const int part = item / groups, g = item - part * groups;
        const int x = (int)lv[g * 32 + lane];
        int r = 0;
#pragma unroll 4
        for (int c = part; c < groups; c += parts) {
            const int *sv = sorted + c * 32;
            const int t = c < g ? x - 1 : x;               // earlier entries count when equal
            int pos = 0;
#pragma unroll
            for (int s = 16; s >= 1; s >>= 1) pos += sv[pos + s - 1] > t ? s : 0;
            r += c == g ? 0 : pos + (sv[pos] > t ? 1 : 0);
        }
        if (r) atomicAdd(rank + g * 32 + lane, r);
    }
    __syncthreads();
    for (int i = tid; i < m; i += NT) {
        const int r = rank[i];
        if (r < CAND) {
            cum[r] = __uint_as_float(lv[i]);
            sid[r] = ids ? (int)ids[i] : i;
        }
    }
    __syncthreads();
}

// Given hist[0..nbins) (nbins <= 2048, non-negative, total below 2^31), find the highest bin d whose suffix sum
// S(d) = hist[d] + hist[d+1] + ... reaches `need` (need >= 1): returns d in every thread, with `above` = S(d+1) and
// `in_bin` = hist[d], or -1 when all bins together do not.  Thread t scans the bins in descending order, 2048 / NT per
// thread; one warp scan, one barrier, a second scan over the warp totals.
template <int NT>
__device__ __forceinline__ int find_suffix_crossing(const int *hist, int nbins, int need, SCShared &sh, int &above,
                                                    int &in_bin)
{
    constexpr int PER = HIST / NT, NW = NT / 32;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    int c[PER], local = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int r = PER * tid + i;                               // rank from the top
        c[i] = r < nbins ? hist[nbins - 1 - r] : 0;
        local += c[i];
    }
    int incl = local;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += x;
    }
    if (lane == 31) sh.red_i[0][w] = incl;
    __syncthreads();
    const int wt = lane < NW ? sh.red_i[0][lane] : 0;
    int wincl = wt;                                                // inclusive scan of the warp totals
#pragma unroll
    for (int o = 1; o < NW; o <<= 1) {
        const int x = __shfl_up_sync(FULL, wincl, o);
        if (lane >= o) wincl += x;
    }
    if (__shfl_sync(FULL, wincl, NW - 1) < need) return -1;
    int excl = __shfl_sync(FULL, wincl - wt, w) + incl - local;
    if (excl < need && need <= excl + local) {
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            if (excl < need && need <= excl + c[i]) {
                sh.bcast_i[4] = nbins - 1 - (PER * tid + i);
                sh.bcast_i[5] = excl;
                sh.bcast_i[6] = c[i];
            }
            excl += c[i];
        }
    }
    __syncthreads();
    above = sh.bcast_i[5];
    in_bin = sh.bcast_i[6];
    return sh.bcast_i[4];
}

// Count into hist[digit] the entries that `match`, one shared-memory atomic per entry; when every matching lane of
// a warp has the same digit (heavily tied data) the warp adds its count with a single atomic instead.
__device__ __forceinline__ void hist_add(int *hist, bool match, unsigned digit, int amount = 1)
{
    const unsigned who = __ballot_sync(FULL, match);
    if (who == 0) return;
    const int leader = __ffs(who) - 1;
    const unsigned d0 = __shfl_sync(FULL, digit, leader);
    const unsigned same = __ballot_sync(FULL, match && digit == d0);
    if (same == who && amount == 1) {
        if ((int)(threadIdx.x & 31) == leader) atomicAdd(&hist[d0], __popc(who));
    } else if (match) {
        atomicAdd(&hist[digit], amount);
    }
}
template <int NT>
__device__ __forceinline__ void hist_clear(int *hist)
{
#pragma unroll
    for (int i = 0; i < HIST / NT; ++i) hist[threadIdx.x + i * NT] = 0;
}

// A bit pattern `thr` with at least CAND and, ties permitting, at most LIST of vals[0..n) (shared memory, values >= 0;
// CAND < n) at or above it, and their number n_ge, by a radix search: digits of 11, 11 and 9 bits from the top, each a
// histogram in shared memory (integer atomics) and a scan for the bin that holds the CAND-th entry.  A pass only
// counts the entries that fell into the previous pass's bin.  After the last pass thr is the CAND-th largest entry.
template <int NT>
__device__ __forceinline__ void radix_threshold(const float *vals, int n, int nk, int *hist, SCShared &sh, unsigned &thr,
                                                int &n_ge)
{
    const int tid = threadIdx.x;
    unsigned prefix = 0;
    int need = CAND, above_total = 0;
#pragma unroll 1
    for (int pass = 0; pass < 3; ++pass) {
        const int shift = pass == 0 ? 20 : (pass == 1 ? 9 : 0);
        const int nbins = pass == 2 ? 512 : 2048;
        const int up = pass == 0 ? 31 : (pass == 1 ? 20 : 9);        // bits at and above `up` are decided
        hist_clear<NT>(hist);
        __syncthreads();
#pragma unroll 1
        for (int k = 0; k < nk; ++k) {
            const int b = k * NT + tid;
            const unsigned x = b < n ? __float_as_uint(vals[b]) : 0u;
            const bool match = b < n && (pass == 0 || (x >> up) == (prefix >> up));
            hist_add(hist, match, (x >> shift) & (unsigned)(nbins - 1));
        }
        __syncthreads();
        int above, in_bin;
        const int d = find_suffix_crossing<NT>(hist, nbins, need, sh, above, in_bin);
        prefix |= (unsigned)d << shift;
        above_total += above;
        need -= above;
        thr = prefix;
        n_ge = above_total + in_bin;
        if (n_ge <= LIST || pass == 2) return;
        __syncthreads();          // hist and the broadcast words are rewritten by the next pass
    }
}

// The min(CAND, n) largest (value, lower-index-first) entries of vals[0..n) (shared memory, values >= 0) in order: values
// to cum[], zero beyond the last, blocks to sid[].  list: 2 * LIST words; counts: nk * NT / 32 words; hist: HIST words.
template <int NT>
__device__ __forceinline__ void select_top_sorted(float *vals, int n, int nk, unsigned *list, int *counts, int *hist, float *cum,
                                                  int *&sid, SCShared &sh)
{
    constexpr int NW = NT / 32;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    sid = hist + LIST;
    if (n <= LIST) {
        for (int i = tid; i < LIST; i += NT) {
            if (i < CAND) cum[i] = 0.0f;
            list[i] = i < n ? __float_as_uint(vals[i]) : 0u;
            hist[i] = 0;
        }
        __syncthreads();
        order_list<NT>(list, nullptr, n, hist, hist + LIST + CAND, cum, sid);
        return;
    }
    unsigned *lv = list, *li = list + LIST;
    unsigned thr = 0u;
    int n_ge = n;            // entries >= thr
    radix_threshold<NT>(vals, n, nk, hist, sh, thr, n_ge);
    // All of them go to the list, in block order.  Where they do not fit, thr is the value of the CAND-th largest entry
    // and many entries equal it: take everything above, then the lowest block ids among the equal.
    const bool ties = n_ge > LIST;
    const unsigned least = ties ? thr + 1u : thr;
#pragma unroll 1
    for (int k = 0; k < nk; ++k) {
        const int b = k * NT + tid;
        const unsigned who = __ballot_sync(FULL, b < n && __float_as_uint(vals[b < n ? b : 0]) >= least);
        if (lane == 0) counts[k * NW + w] = __popc(who);
    }
    __syncthreads();             // the histogram has been read as well
    for (int i = tid; i < LIST; i += NT) { lv[i] = 0u; hist[i] = 0; }
    __syncthreads();
    int base = 0;
#pragma unroll 1
    for (int k = 0; k < nk; ++k) {
        const int b = k * NT + tid;
        const int cw = lane < NW ? counts[k * NW + lane] : 0;
        const int before = __reduce_add_sync(FULL, lane < w ? cw : 0), total = __reduce_add_sync(FULL, cw);
        const unsigned x = b < n ? __float_as_uint(vals[b]) : 0u;
        const unsigned who = __ballot_sync(FULL, b < n && x >= least);
        if ((who >> lane) & 1u) {
            const int pos = base + before + __popc(who & ((1u << lane) - 1u));
            lv[pos] = x;
            li[pos] = (unsigned)b;
        }
        base += total;
    }
    int m = base;
    if (ties) {
        // entries equal to the threshold fill the remaining places in block order, NT consecutive blocks per round
        int par = 0;
        for (int b0 = 0; b0 < n && m < CAND; b0 += NT) {
            const int b = b0 + tid;
            const bool eq = b < n && __float_as_uint(vals[b]) == thr;
            const unsigned who = __ballot_sync(FULL, eq);
            if (lane == 0) sh.red_i[par][w] = __popc(who);
            __syncthreads();
            const int cw = lane < NW ? sh.red_i[par][lane] : 0;
            par ^= 1;
            const int before = __reduce_add_sync(FULL, lane < w ? cw : 0), total = __reduce_add_sync(FULL, cw);
            const int pos = m + before + __popc(who & ((1u << lane) - 1u));
            if (eq && pos < CAND) { lv[pos] = thr; li[pos] = (unsigned)b; }
            m += total;
        }
        m = min(m, CAND);
    }
    __syncthreads();
    order_list<NT>(lv, li, m, hist, hist + LIST + CAND, cum, sid);
}

// The four largest (value, lower index first) of a warp's lanes, each lane holding a descending list of four (padding:
// value 0): four rounds of a warp-wide maximum over the list heads; the lane that wins pops its list.
struct Top4 {
    unsigned v[4], i[4];
};
__device__ __forceinline__ void warp_top4(Top4 &t, Top4 &out)
{
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const unsigned best = __reduce_max_sync(FULL, t.v[0]);
        const unsigned idx = __reduce_min_sync(FULL, t.v[0] == best ? t.i[0] : 0xFFFFFFFFu);
        out.v[r] = best;
        out.i[r] = idx;
        if (t.v[0] == best && t.i[0] == idx) {
#pragma unroll
            for (int j = 0; j < 3; ++j) { t.v[j] = t.v[j + 1]; t.i[j] = t.i[j + 1]; }
            t.v[3] = 0u;
            t.i[3] = 0xFFFFFFFFu;
        }
    }
}

// "Column sums" of the value check for up to three admission thresholds at once: of the entries e[0..n) (shared
// memory), column t (0..1023) adds its admitted members t, t + 1024, ... in ascending order; 32 neighbouring columns
// are combined by the butterfly 16,8,4,2,1 and the 32 sums of that by the same butterfly.  f[i] = sum of the entries
// with bits >= t[i], c[i] = their number; results in every thread.  Adding an admitted entry never lowers a sum (every
// step is a monotone rounding), which is what the threshold search relies on.  A threshold of 0xFFFFFFFF admits nothing.
template <int NT>
__device__ __forceinline__ void column_sums3(const float *e, int n, unsigned t1, unsigned t2, unsigned t3, SCShared &sh,
                                             int &parity, float (&f)[3], int (&c)[3])
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll 1
    for (int g = w; g < 32; g += NT / 32) {
        float s1 = 0.0f, s2 = 0.0f, s3 = 0.0f;
        unsigned n12 = 0, n3 = 0;
#pragma unroll 1
        for (int b = g * 32 + lane; b - lane < n; b += 1024) {
            if (b < n) {
                const float v = e[b];
                const unsigned x = __float_as_uint(v);
                if (x >= t1) { s1 = __fadd_rn(s1, v); n12 += 1u; }
                if (x >= t2) { s2 = __fadd_rn(s2, v); n12 += 1u << 16; }
                if (x >= t3) { s3 = __fadd_rn(s3, v); n3 += 1u; }
            }
        }
        if (g * 32 < n) {
            s1 = warp_sum(s1);
            s2 = warp_sum(s2);
            s3 = warp_sum(s3);
            n12 = __reduce_add_sync(FULL, n12);
            n3 = __reduce_add_sync(FULL, n3);
        }
        if (lane == 0) {
            sh.red_f3[parity][0][g] = s1;
            sh.red_f3[parity][1][g] = s2;
            sh.red_f3[parity][2][g] = s3;
            sh.red_u[parity][0][g] = n12;
            sh.red_u[parity][1][g] = n3;
        }
    }
    __syncthreads();
    f[0] = warp_sum(sh.red_f3[parity][0][lane]);
    f[1] = warp_sum(sh.red_f3[parity][1][lane]);
    f[2] = warp_sum(sh.red_f3[parity][2][lane]);
    const unsigned c12 = __reduce_add_sync(FULL, sh.red_u[parity][0][lane]);
    c[2] = (int)__reduce_add_sync(FULL, sh.red_u[parity][1][lane]);
    c[0] = (int)(c12 & 0xFFFFu);
    c[1] = (int)(c12 >> 16);
    parity ^= 1;
}

// One column sum (same order as column_sums3) over the entries that `admit` (bits, block id) takes.
template <int NT, typename F>
__device__ __forceinline__ float column_sum1(const float *e, int n, SCShared &sh, int &parity, int &count, F admit)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll 1
    for (int g = w; g < 32; g += NT / 32) {
        float s = 0.0f;
        unsigned c = 0;
#pragma unroll 1
        for (int b = g * 32 + lane; b - lane < n; b += 1024) {
            if (b < n) {
                const float v = e[b];
                if (admit(__float_as_uint(v), b)) { s = __fadd_rn(s, v); ++c; }
            }
        }
        if (g * 32 < n) {
            s = warp_sum(s);
            c = __reduce_add_sync(FULL, c);
        }
        if (lane == 0) { sh.red_f3[parity][0][g] = s; sh.red_u[parity][0][g] = c; }
    }
    __syncthreads();
    const float r = warp_sum(sh.red_f3[parity][0][lane]);
    count = (int)__reduce_add_sync(FULL, sh.red_u[parity][0][lane]);
    parity ^= 1;
    return r;
}

template <typename T2>
__device__ __forceinline__ void rescore_block(const cqa_cache &c, const void *q, int q_dtype, int h, long bid,
                                              long n_scoring_tokens, float q_scale, float &s, float &lm, const float *q_row)
{
    fp16_block_score_warp<T2>(c, q, q_dtype, h, bid, n_scoring_tokens, q_scale, s, lm, q_row);
}
// First row of Tier-2 key block `bid`, or NULL when neither tier holds it.
__device__ __forceinline__ const char *t2_block_any(const cqa_cache &c, int kv, long bid)
{
    if (c.t2_dtype == CQA_BF16) return reinterpret_cast<const char *>(t2_key_block<__nv_bfloat16>(c, kv, bid));
    if (c.t2_dtype == CQA_F16) return reinterpret_cast<const char *>(t2_key_block<__half>(c, kv, bid));
    return reinterpret_cast<const char *>(t2_key_block<float>(c, kv, bid));
}
// The logits of N tokens, by the 16 lanes of a half warp each (same arithmetic as fp16_block_score_warp); all rows are
// requested before the first is used.
template <int N, typename T2>
__device__ __forceinline__ void token_logits_t(const void *const (&row)[N], const float *q_row, float q_scale, float (&lg)[N])
{
    const int L = threadIdx.x & 15;
    Raw8<T2> raw[N];
#pragma unroll
    for (int i = 0; i < N; ++i) raw[i] = row[i] ? raw_load8<T2>(reinterpret_cast<const T2 *>(row[i])) : raw_zero8<T2>();
    float qv[8];
    load8<float>(q_row + 8 * L, qv);
#pragma unroll
    for (int i = 0; i < N; ++i) {
        float kf[8];
        raw_to_f(raw[i], kf);
        const float d = hw_sum(chain8(kf, qv));
        lg[i] = row[i] ? __fmul_rn(d, q_scale) : -INFINITY;
    }
}
template <int N>
__device__ __forceinline__ void token_logits(const cqa_cache &c, const void *const (&row)[N], const float *q_row, float q_scale, float (&lg)[N])
{
    if (c.t2_dtype == CQA_BF16) token_logits_t<N, __nv_bfloat16>(row, q_row, q_scale, lg);
    else if (c.t2_dtype == CQA_F16) token_logits_t<N, __half>(row, q_row, q_scale, lg);
    else token_logits_t<N, float>(row, q_row, q_scale, lg);
}

// Tier-2 dtype dispatch at run time: the re-score is a few warps of one role, the rest of the kernel does not
// depend on the dtype.
__device__ __noinline__ void rescore_block_any(const cqa_cache &c, const void *q, int q_dtype, int h, long bid,
                                               long n_scoring_tokens, float q_scale, float &s, float &lm,
                                               const float *q_row)
{
    if (c.t2_dtype == CQA_BF16) rescore_block<__nv_bfloat16>(c, q, q_dtype, h, bid, n_scoring_tokens, q_scale, s, lm, q_row);
    else if (c.t2_dtype == CQA_F16) rescore_block<__half>(c, q, q_dtype, h, bid, n_scoring_tokens, q_scale, s, lm, q_row);
    else rescore_block<float>(c, q, q_dtype, h, bid, n_scoring_tokens, q_scale, s, lm, q_row);
}

// Dynamic shared memory: A[n_arr] B[n_arr] C[n_pad] (floats; n_arr = max(n_pad, 2048)), list[2 * LIST], cum[CAND],
// gsum, leaf, mask[n_pad] (bytes).  The full-sort fallback aliases its keys over A and B; the radix searches use the
// array that is free at that point as their histogram.
template <int NT>
__device__ __forceinline__ void selcert_body(const cqa_cache &c, const cqa_knobs &kn, const cqa_workspace &ws, const void *q,
                                             int q_dtype, long nq, long nact, const float *u, long u_ld, int n_pad, int hi,
                                             int base_width, int two_level, int rk, int phases, int role_base)
{
    extern __shared__ __align__(16) unsigned char dsm[];
    const int n_arr = n_pad > 2048 ? n_pad : 2048;
    float *A = reinterpret_cast<float *>(dsm);                 // m_b; role 2 later: contributions mass * eta
    float *B = A + n_arr;                                      // S_b; then mass / block log-mass / histogram
    float *C = B + n_arr;                                      // uniforms or eta_b; then mass fractions / histogram
    unsigned *list = reinterpret_cast<unsigned *>(C + n_pad);
    float *cum = reinterpret_cast<float *>(list + 2 * LIST);
    float *gsum = cum + CAND;
    float *leaf = gsum + ((n_pad > 1024 ? n_pad : 1024) >> 5);
    unsigned char *mask = reinterpret_cast<unsigned char *>(leaf + (n_pad >> 8) + 8);
    constexpr int NW = NT / 32;
    __shared__ SCShared sh;
    __shared__ int top_idx[CQA_MAX_RANKING_K];
    __shared__ float top_i8[CQA_MAX_RANKING_K], top_f16[CQA_MAX_RANKING_K], top_lm[CQA_MAX_RANKING_K];
    __shared__ float s_delta;
    __shared__ __align__(16) float s_q[D];           // role 1: the head's query row as floats
    __shared__ unsigned s_topv[NW * 4], s_topi[NW * 4];
    __shared__ float s_lg[4 * BS];     // role 1: token logits of the candidates

    __shared__ __align__(8) uint64_t row_bar;
    if (threadIdx.x == 0) {
        mbar_init(&row_bar, 1);
        mbar_init_fence();
    }
    __syncthreads();   // before the wait on the previous kernel: this part overlaps its tail

    const int h = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kv = h / c.gqa_group;
    const int n = (int)nq;
    const int nk = (n + NT - 1) / NT;                          // blocks per thread: b = k * NT + tid, k < nk
    // Plain layout: row h of an [H][ld] array.  Sharded layout: row h of rank r's slot in the all-gather buffer,
    // [rank][row][chunk]; global block b sits at rank r = min(b / stride, ranks - 1), column b - r * stride.
    const bool sharded_in = ws.shard_stride > 0;
    const long row_ld = sharded_in ? ws.shard_chunk : ws.ld;
    const float *mb = ws.m_b + (long)h * row_ld;
    const float *sb = ws.s_b + (long)h * row_ld;
    // 32-bit arithmetic on purpose: the mapping runs once per block and thread
    const int sh_stride = sharded_in ? (int)ws.shard_stride : 1, sh_last = ws.shard_ranks - 1;
    const long sh_rank_stride = ws.shard_rank_stride;
    float *mf = ws.mass_frac + (long)h * ws.ld;
    cqa_head_cert *ct = ws.cert + h;
    // Three independent roles per head run as separate CTAs (grid.y): 0 = selector, 1 = ranking /
    // boundary / consistency checks, 2 = value check.  Roles 0 and 2 both need the mass fractions and
    // compute them with the same canonical arithmetic, so no CTA waits for another.
    const int role = role_base + (int)blockIdx.y;
    const bool fused = (phases & PH_SELECT) != 0;
    const bool compute_frac = role == 0 || (role == 2 && fused);
    const bool have_int4 = c.values_int4_packed != nullptr && c.values_int4_errors != nullptr;
    int parity = 0;

    // ---- the rows go from global to shared memory without passing through registers:
    // A <- m_b, B <- S_b, C <- eta_b (role 2) or the exploration uniforms (role 0)
    const bool explore_on = role == 0 && kn.exploration_rate > 0.0f;
    const float *eta = have_int4 ? c.values_int4_errors + (long)kv * (sharded_in ? ws.shard_chunk : c.max_blocks) : nullptr;
    const bool frac_given = role == 2 && !fused;
    const float *xsrc = role == 2 ? eta : ((explore_on && u != nullptr) ? u + (long)h * u_ld : nullptr);
    // Rows that start on a 16-byte boundary are fetched by the bulk-copy engine: one thread issues the copies (one
    // per array, or one per array and rank in the sharded layout, whose per-rank pieces are contiguous) and every
    // thread waits on the barrier they report to (bounded).  The last n % 4 blocks and unaligned rows go by 4-byte
    // asynchronous copies, each thread copying the blocks it owns.
    const float *bsrc = frac_given ? mf : sb;
    const int n4 = n & ~3;
    const int nseg = sharded_in ? ws.shard_ranks : 1;
    const int last_first = (nseg - 1) * sh_stride;             // first block of the last piece
    const bool pieces_ok = !sharded_in || (((sh_stride | (int)(sh_rank_stride & 0x7fffffff)) & 3) == 0 && n > last_first);
    const bool bulk = pieces_ok && n4 > 0 &&
                      (((uintptr_t)mb | (uintptr_t)bsrc | (uintptr_t)(xsrc ? xsrc : mb)) & 15u) == 0;
    // Still nothing of the previous kernel has been read: the exploration bits depend on the seed alone and are drawn
    // while that kernel drains.  One Philox call gives the eight 16-bit uniforms of blocks tid + 1024 * (8j .. 8j+7).
    const bool drawn = explore_on && u == nullptr;
    if (drawn) {
        const int nkp = n_pad > 1024 ? n_pad / 1024 : 1;
#pragma unroll 1
        for (int col = tid; col < 1024 && col < n_pad; col += NT) {
#pragma unroll 1
            for (int j = 0; j * 8 < nkp; ++j) {
                const uint4 r = philox4(ws.rng_seed, ws.rng_offset, (unsigned)h, (unsigned)col | ((unsigned)j << 10));
                const unsigned wds[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int b = (8 * j + i) * 1024 + col;
                    if (8 * j + i < nkp && b < n_pad) {
                        const float uni = (float)((wds[i >> 1] >> ((i & 1) * 16)) & 0xFFFFu) * 1.52587890625e-05f;   // 2^-16
                        mask[b] = (b < n && uni < kn.exploration_rate) ? 2 : 0;   // bit 1: exploration candidate
                    }
                }
            }
        }
    }

    // Role 1, also ahead of the wait: the query row and Delta depend on q and on the per-channel scale maxima, both
    // complete before the score kernel started (the scale maxima of a sharded run arrive with the exchange and are
    // read after it).  The re-scoring warps later find q in shared memory and have one round trip to DRAM less.
    const bool rank_checks = role == 1 && (kn.ranking_fallback || kn.score_consistency) && n > 0 && q != nullptr;
    const bool delta_early = rank_checks && !sharded_in && !(phases & PH_TOP_ONLY) && c.sigma_max != nullptr;
    if (rank_checks) {
        if (warp == 0)
            for (int i = lane; i < D; i += 32) s_q[i] = load_q(q, q_dtype, (long)h * D + i);
        if (warp == 1 && delta_early) {
            const float d = delta_bound_warp(c, q, q_dtype, h);
            if (lane == 0) s_delta = d;
        }
    }

    grid_dependency_wait();
    peer_wait(ws.wait_flags, ws.wait_n, ws.wait_skip, ws.wait_value, ws.wait_status, 1, ws.wait_spins);

    if (bulk && tid == 0) {
        const unsigned bar = smem_u32(&row_bar);
        mbar_arrive_expect_tx(bar, (unsigned)n4 * 4u * (xsrc ? 3u : 2u));
#pragma unroll 1
        for (int r = 0; r < nseg; ++r) {
            const int first = r * sh_stride;
            const int cnt = (r == nseg - 1 ? n4 : first + sh_stride) - first;     // blocks of this piece, a multiple of 4
            if (cnt <= 0) continue;
            const long go = sharded_in ? (long)r * sh_rank_stride : 0;
            const unsigned bytes = (unsigned)cnt * 4u;
            bulk_copy_g2s(smem_u32(A + first), mb + go, bytes, bar);
            bulk_copy_g2s(smem_u32(B + first), frac_given ? mf + first : sb + go, bytes, bar);
            if (xsrc) bulk_copy_g2s(smem_u32(C + first), role == 2 ? xsrc + go : xsrc + first, bytes, bar);
        }
    }
#pragma unroll 1
    for (int k = bulk ? n4 / NT : 0; k < nk; ++k) {
        const int b = k * NT + tid;
        if (b < n && !(bulk && b < n4)) {
            long gb = b;
            if (sharded_in) {
                int r = b / sh_stride;
                if (r > sh_last) r = sh_last;
                gb = (long)r * sh_rank_stride + (b - r * sh_stride);
            }
            cp_async4(A + b, mb + gb);
            // certifying only: the mass fractions were computed by the selector call and take the place of S_b
            cp_async4(B + b, frac_given ? mf + b : sb + gb);
            if (xsrc) cp_async4(C + b, xsrc + (role == 2 ? gb : (long)b));
        }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    if (bulk) mbar_wait(smem_u32(&row_bar), 0u);
    // each thread reads back only what it copied itself until the next barrier

    // ---- per-block preparation: the head's largest m_b; exploration bits (role 0); block log-masses (role 1)
    float mg = -INFINITY;
    if (role == 0) {
#pragma unroll 1
        for (int k = 0; k < nk; ++k) {
            const int b = k * NT + tid;
            if (b < n_pad) {
                if (!drawn)   // bit 1: exploration candidate (uniforms given by the caller), bit 0: selected (set later)
                    mask[b] = (explore_on && b < n && C[b] < kn.exploration_rate) ? 2 : 0;
                if (b < n) mg = fmaxf(mg, A[b]);
            }
        }
    } else {
#pragma unroll 1
        for (int k = 0; k < nk; ++k) {
            const int b = k * NT + tid;
            if (b < n) {
                const float m = A[b];
                mg = fmaxf(mg, m);
                if (role == 1) B[b] = __fadd_rn(clog(fmaxf(B[b], 1e-30f)), m);   // block log-mass for the boundary check
            }
        }
    }
    float total = 0.0f;
    if (compute_frac) {
        // mass = S * exp(m - max m) into B, fraction = mass * (1 / total): role 0 into C (and global memory),
        // role 2 straight into the contributions
        mg = cta_max<NT>(mg, sh, parity);
#pragma unroll 1
        for (int k = 0; k < nk; ++k) {
            const int b = k * NT + tid;
            if (b < n) B[b] = __fmul_rn(fmaxf(B[b], 1e-30f), cexp(__fsub_rn(A[b], mg)));
        }
        total = fmaxf(cta_canonical_sum<NT>(B, n, nk, gsum, leaf), 1e-30f);
        const float inv_total = __fdiv_rn(1.0f, total);
#pragma unroll 1
        for (int k = 0; k < nk; ++k) {
            const int b = k * NT + tid;
            if (b < n) {
                const float f = __fmul_rn(B[b], inv_total);
                if (role == 0) { C[b] = f; mf[b] = f; }
                else A[b] = __fmul_rn(f, C[b]);           // role 2: contribution = mass fraction * eta_b
            }
        }
    } else if (role == 2) {
#pragma unroll 1
        for (int k = 0; k < nk; ++k) {
            const int b = k * NT + tid;
            if (b < n) A[b] = __fmul_rn(B[b], C[b]);
        }
    }
    __syncthreads();

    if (role == 0) {
        // the `hi` heaviest blocks, sorted
        int32_t *sidx = ws.sorted_idx + (long)h * ws.sel_width;
        float *scum = ws.sorted_cumsum + (long)h * ws.sel_width;
        const bool narrow = hi <= CAND;
        int *sid = nullptr;
        unsigned char *tm = ws.topk_mask + (long)h * ws.ld;
        unsigned char *em = ws.explore_mask + (long)h * ws.ld;
        // Exploration candidates of all blocks to global memory, as if K* selected none of them (corrected below), by
        // threads t0, t0 + 1, ...: four blocks per store when the rows allow it (mask[] is 4-byte aligned, n_pad a
        // multiple of 32).
        const auto write_masks = [&](int t0) {
            int explored = 0;
            const int n4w = ((((uintptr_t)tm | (uintptr_t)em) & 3u) == 0) ? (n & ~3) : 0;
            const unsigned *mask4 = reinterpret_cast<const unsigned *>(mask);
#pragma unroll 1
            for (int b = 4 * (tid - t0); b < n4w; b += 4 * (NT - t0)) {
                const unsigned exp = (mask4[b >> 2] >> 1) & 0x01010101u;
                explored += __popc(exp);
                *reinterpret_cast<unsigned *>(tm + b) = exp;
                *reinterpret_cast<unsigned *>(em + b) = exp;
            }
#pragma unroll 1
            for (int b = n4w + tid - t0; b < (int)nact; b += NT - t0) {
                const unsigned char e = b < n ? (mask[b] >> 1) & 1 : 0;
                explored += e;
                tm[b] = b < n ? e : 1;
                em[b] = e;
            }
            explored = __reduce_add_sync(FULL, explored);
            if (lane == 0 && explored) atomicAdd(&sh.counter2, explored);
        };
        if (tid == 0) sh.counter2 = 0;
        if (narrow) {
            select_top_sorted<NT>(C, n, nk, list, reinterpret_cast<int *>(gsum), reinterpret_cast<int *>(B), cum, sid, sh);
            if (tid == 0) {
                // sequential prefix sum in place; the next 32 values are fetched while 32 are added, so that only the
                // additions are serial
                float run = 0.0f;
                float4 *c4 = reinterpret_cast<float4 *>(cum);
                float4 v[8], nx[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) nx[i] = c4[i];
#pragma unroll 1
                for (int j0 = 0; j0 < hi; j0 += 32) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) v[i] = nx[i];
                    if (j0 + 32 < CAND) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) nx[i] = c4[(j0 >> 2) + 8 + i];
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        v[i].x = (j0 == 0 && i == 0) ? v[i].x : __fadd_rn(run, v[i].x);
                        v[i].y = __fadd_rn(v[i].x, v[i].y);
                        v[i].z = __fadd_rn(v[i].y, v[i].z);
                        v[i].w = __fadd_rn(v[i].z, v[i].w);
                        run = v[i].w;
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i) c4[(j0 >> 2) + i] = v[i];
                }
            } else if (tid >= 32) {
                for (int j = tid - 32; j < hi; j += NT - 32) sidx[j] = sid[j];
                write_masks(32);
            }
        } else {
            // wide selections (k_max unset or very large): full sort, prefix sums straight to global memory
            __syncthreads();
            write_masks(0);
            u64 *keys = reinterpret_cast<u64 *>(A);   // m_b and the masses are not needed any more
            for (int b = tid; b < n_pad; b += NT) keys[b] = b < n ? make_key(C[b], b) : 0ull;
            __syncthreads();
            bitonic_sort_desc<NT>(keys, n_pad);
            if (tid == 0) {
                float run = 0.0f;
                for (int j = 0; j < hi; ++j) {
                    const float v = key_val(keys[j]);
                    run = j == 0 ? v : __fadd_rn(run, v);
                    scum[j] = run;
                    sidx[j] = key_idx(keys[j]);
                }
            }
        }
        __syncthreads();
        // K*, Rung 1: the prefix sums are non-decreasing, so the first index with cum >= tau is the number of entries
        // below tau; every thread works K* out for itself
        const float *cs = narrow ? cum : scum;
        int ss = 0;
        if (hi <= NT) {
            ss = __syncthreads_count(tid < hi && cs[tid < hi ? tid : 0] < kn.tau_cov);
        } else {
            int below = 0;
            for (int j = tid; j < hi; j += NT) below += cs[j] < kn.tau_cov ? 1 : 0;
            if (tid == 0) sh.counter = 0;
            __syncthreads();
            if (below) atomicAdd(&sh.counter, below);
            __syncthreads();
            ss = sh.counter;
            __syncthreads();
        }
        const int k_e = min(max(ss + 1, min(kn.k_min, hi)), hi);
        const float ta_e = cs[k_e - 1];
        const float tl_e = fmaxf(__fsub_rn(1.0f, ta_e), 0.0f);
        int k_star = k_e, trig = 0, k_b = k_e;
        float ta = ta_e, tl = tl_e;
        if (two_level) {
            k_b = min(max(min(ss, base_width) + 1, min(kn.k_min, base_width)), base_width);
            const float ta_b = cs[k_b - 1];
            const float tl_b = fmaxf(__fsub_rn(1.0f, ta_b), 0.0f);
            trig = tl_b > kn.rung1_threshold ? 1 : 0;
            if (!trig) { k_star = k_b; ta = ta_b; tl = tl_b; }
        } else if (kn.rung1_threshold >= 0.0f && kn.k_max > 0) {
            trig = tl_e > kn.rung1_threshold ? 1 : 0;
        }
        int taken = 0;           // selected blocks that were exploration candidates
        for (int j = tid; j < k_star; j += NT) {
            const int b = narrow ? sid[j] : sidx[j];
            tm[b] = 1;
            if (mask[b]) { em[b] = 0; ++taken; }
        }
        if (narrow)
            for (int j = tid; j < hi; j += NT) scum[j] = cum[j];
        taken = __reduce_add_sync(FULL, taken);
        if (lane == 0 && taken) atomicAdd(&sh.counter2, -taken);
        if (tid == 0) {
            ct->k_star = k_star;
            ct->k_star_base = k_b;
            ct->k_star_expanded = k_e;
            ct->rung1_triggered = trig;
            ct->tail_mass = tl;
            ct->tau_actual = ta;
            ct->m_global = mg;
            ct->total_mass = total;
            if (trig) atomicOr(ws.any_flags + 0, 1);
        }
        __syncthreads();
        if (tid == 0) ct->exploration_blocks = sh.counter2;
        return;
    }

    // ---- ranking / boundary / score consistency
    const bool need_fp16 = (kn.ranking_fallback || kn.score_consistency) && n > 0;
    if (role == 1 && need_fp16) {
        const bool given = (phases & PH_GIVEN) != 0;
        if (given) {
            if (tid < rk) {
                const int b = ct->top_blocks[tid];
                top_idx[tid] = b;
                if (b >= 0) B[b] = -INFINITY;
                top_i8[tid] = A[b];
                // one array per rank when the re-scores were pushed (only a block's owner wrote non-zero values)
                float gs = 0.0f, gl = 0.0f;
                const int gr = ws.given_ranks > 1 ? ws.given_ranks : 1;
                for (int r = 0; r < gr; ++r) {
                    const float *g = ws.given_fp16 + r * ws.given_rank_stride + ((long)h * CQA_MAX_RANKING_K + tid) * 2;
                    gs = __fadd_rn(gs, g[0]);
                    gl = __fadd_rn(gl, g[1]);
                }
                top_f16[tid] = gs;
                top_lm[tid] = gl;
            }
        } else if (rk <= 4) {
            Top4 t4, w4;
#pragma unroll
            for (int i = 0; i < 4; ++i) { t4.v[i] = 0u; t4.i[i] = 0xFFFFFFFFu; }
#pragma unroll 1
            for (int k = 0; k < nk; ++k) {
                const int b = k * NT + tid;
                unsigned v = b < n ? orderable(A[b]) : 0u, id = (unsigned)b;
                if (__any_sync(FULL, v > t4.v[3])) {
                    // descending insertion; blocks come in ascending order, so among equal ones the earlier stays ahead
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const bool gt = v > t4.v[i];
                        const unsigned hv = gt ? v : t4.v[i], hi_ = gt ? id : t4.i[i];
                        v = gt ? t4.v[i] : v;
                        id = gt ? t4.i[i] : id;
                        t4.v[i] = hv;
                        t4.i[i] = hi_;
                    }
                }
            }
            warp_top4(t4, w4);
            if (lane == 0) {
#pragma unroll
                for (int i = 0; i < 4; ++i) { s_topv[warp * 4 + i] = w4.v[i]; s_topi[warp * 4 + i] = w4.i[i]; }
            }
            __syncthreads();
            if (warp == 0) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    t4.v[i] = lane < NW ? s_topv[lane * 4 + i] : 0u;
                    t4.i[i] = lane < NW ? s_topi[lane * 4 + i] : 0xFFFFFFFFu;
                }
                warp_top4(t4, w4);
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    if (lane == r && r < rk) {
                        top_idx[r] = (int)w4.i[r];
                        top_i8[r] = A[w4.i[r]];
                        B[w4.i[r]] = -INFINITY;           // not part of the boundary maximum
                    }
            }
        } else {
            unsigned pv = 0xFFFFFFFFu, pi = 0u;      // the previous winner: value, block
            for (int r = 0; r < rk; ++r) {
                unsigned bv = 0u, bi = 0xFFFFFFFFu;
                for (int b = tid; b < n; b += NT) {
                    const unsigned v = orderable(A[b]);
                    if ((r == 0 || v < pv || (v == pv && (unsigned)b > pi)) && v > bv) { bv = v; bi = (unsigned)b; }
                }
                const unsigned wv = __reduce_max_sync(FULL, bv);
                const unsigned wi = __reduce_min_sync(FULL, bv == wv ? bi : 0xFFFFFFFFu);
                __syncthreads();
                if (lane == 0) { s_topv[warp] = wv; s_topi[warp] = wi; }
                __syncthreads();
                const unsigned cv = s_topv[lane & (NW - 1)], ci = s_topi[lane & (NW - 1)];
                pv = __reduce_max_sync(FULL, cv);
                pi = __reduce_min_sync(FULL, cv == pv ? ci : 0xFFFFFFFFu);
                if (tid == 0) {
                    top_idx[r] = (int)pi;
                    top_i8[r] = A[pi];
                    B[pi] = -INFINITY;
                }
            }
        }
        __syncthreads();
        if (phases & PH_TOP_ONLY) {
            if (tid < CQA_MAX_RANKING_K) ct->top_blocks[tid] = tid < rk ? top_idx[tid] : -1;
            return;
        }
        // Boundary bound: max over the blocks outside the top list of (ell_b + delta).  Rounding is monotone, so it equals
        // (max ell_b) + delta; the maximum is taken while the Tier-2 rows of the candidates are on their way.
        const bool peer_b = (phases & PH_PEER_B) != 0;
        // With at most four candidates and Delta already known, a candidate block is re-scored by a quarter of the warps
        // (a half warp per token): a single warp walking all 16 tokens is a chain of ~600 dependent instructions behind a
        // DRAM round trip, run once, and was the longest step of this role.
        const bool spread = !given && rk <= 4 && (delta_early || peer_b);
        constexpr int WPC = NW / 4, TPH = BS / (2 * WPC);      // warps per candidate, tokens per half warp
        const int cj = warp / WPC;                             // this warp's candidate
        // sharded by block range: this rank re-scores the candidates it owns (local block ids) and sends zeros for the
        // others, so that the sum over the ranks' rows is the owner's row
        const void *row[TPH] = {};
        if (spread) {
            const long bid = cj < rk ? (long)top_idx[cj] - (peer_b ? ws.peer_first_block : 0) : -1;
            const bool owned = cj < rk && bid >= 0 && (!peer_b || bid < ws.peer_n_local);
            const char *base = owned ? t2_block_any(c, kv, bid) : nullptr;
            const int esz = c.t2_dtype == CQA_F32 ? 4 : 2, first = (warp % WPC) * 2 + (lane >> 4);
            const long left = (peer_b ? ws.peer_n_local : nq) * BS - bid * BS;        // tokens that take part
            if (base) {
#pragma unroll
                for (int i = 0; i < TPH; ++i) {
                    const int t = first + i * 2 * WPC;
                    if (t < left) row[i] = base + (t * D + 8 * (lane & 15)) * esz;
                    if (row[i] && c.key_slots == nullptr) asm volatile("prefetch.global.L2 [%0];" ::"l"(row[i]));   // device memory only
                }
            }
        }
        float ubm = -INFINITY;
        if (kn.ranking_fallback) {
#pragma unroll 1
            for (int b = tid; b < n; b += NT) ubm = fmaxf(ubm, B[b]);
            ubm = warp_max(ubm);
            if (lane == 0) sh.red_f[0][warp] = ubm;
        }
        if (spread) {
            if (cj < rk) {
                float lg[TPH];
                token_logits<TPH>(c, row, s_q, kn.q_scale, lg);
#pragma unroll
                for (int i = 0; i < TPH; ++i)
                    if ((lane & 15) == 0) s_lg[cj * BS + (warp % WPC) * 2 + (lane >> 4) + i * 2 * WPC] = lg[i];
            }
            if (warp == NW - 1 && !delta_early) {
                const float d = delta_bound_warp(c, q, q_dtype, h, sharded_in ? ws.shard_ranks : 1, ws.shard_rank_stride);
                if (lane == 0) s_delta = d;
            }
            __syncthreads();
            if (warp == 0) {
                // a half warp per candidate: maximum and canonical sum over its 16 tokens
#pragma unroll
                for (int j0 = 0; j0 < 4; j0 += 2) {
                    const int j = j0 + (lane >> 4);
                    const float lg = j < rk ? s_lg[j * BS + (lane & 15)] : -INFINITY;
                    const float mx = hw_max(lg);
                    const float l = fmaxf(hw_sum(lg == -INFINITY ? 0.0f : cexp(__fsub_rn(lg, mx))), 1e-30f);
                    const long bid = j < rk ? (long)top_idx[j] - (peer_b ? ws.peer_first_block : 0) : -1;
                    const bool owned = j < rk && (!peer_b || (bid >= 0 && bid < ws.peer_n_local));
                    const float sc = owned ? mx : 0.0f;
                    const float lm = !owned ? 0.0f : (mx == -INFINITY ? -INFINITY : __fadd_rn(mx, clog(l)));
                    if (j < rk) {
                        if (peer_b) {
                            const int p = lane & 15;          // one lane per destination rank
                            if (p < ws.peer_world) {
                                float *d = ws.peer_xb[p] + ((long)h * CQA_MAX_RANKING_K + j) * 2;
                                d[0] = sc;
                                d[1] = lm;
                            }
                        } else if ((lane & 15) == 0) {
                            top_f16[j] = sc;
                            top_lm[j] = lm;
                        }
                    }
                }
                __syncwarp();
            }
        } else {
            // one warp per candidate, Delta by the next
#pragma unroll 1
            for (int i = warp; i <= rk; i += NW) {
                if (i == rk) {
                    if (!delta_early) {
                        const float d = delta_bound_warp(c, q, q_dtype, h, sharded_in ? ws.shard_ranks : 1, ws.shard_rank_stride);
                        if (lane == 0) s_delta = d;
                    }
                } else if (peer_b) {
                    // re-score the block if this rank owns it (local block ids), zeros otherwise; every rank gets the row
                    const long bl = (long)top_idx[i] - ws.peer_first_block;
                    float s = 0.0f, lm = 0.0f;
                    if (bl >= 0 && bl < ws.peer_n_local)
                        rescore_block_any(c, q, q_dtype, h, bl, ws.peer_n_local * BS, kn.q_scale, s, lm, s_q);
                    if (lane < ws.peer_world) {
                        float *d = ws.peer_xb[lane] + ((long)h * CQA_MAX_RANKING_K + i) * 2;
                        d[0] = s;
                        d[1] = lm;
                    }
                } else if (!given) {
                    float s, lm;
                    rescore_block_any(c, q, q_dtype, h, (long)top_idx[i], nq * BS, kn.q_scale, s, lm, s_q);
                    if (lane == 0) { top_f16[i] = s; top_lm[i] = lm; }
                }
            }
        }
        // in the spread form warp 0 alone goes on to the flags, with what it wrote itself
        if (peer_b || !spread) __syncthreads();
        if (peer_b) {
            // publish this rank's rows of head h, then wait (bounded) for the other ranks' rows and add them up
            if (tid == 0) {
                __threadfence_system();
                for (int p = 0; p < ws.peer_world; ++p)
                    if (p != ws.peer_rank)
                        st_release_sys(ws.peer_flags_b[p] + (long)ws.peer_rank * gridDim.x + h, ws.peer_step);
            }
            peer_wait(ws.peer_flags_b[ws.peer_rank] + h, ws.peer_world, ws.peer_rank, ws.peer_step, ws.wait_status,
                      (long)gridDim.x, ws.wait_spins);
            if (tid < rk) {
                float gs = 0.0f, gl = 0.0f;
                for (int r = 0; r < ws.peer_world; ++r) {
                    const float *g = ws.given_fp16 + r * ws.given_rank_stride + ((long)h * CQA_MAX_RANKING_K + tid) * 2;
                    gs = __fadd_rn(gs, __ldcg(g));
                    gl = __fadd_rn(gl, __ldcg(g + 1));
                }
                top_f16[tid] = gs;
                top_lm[tid] = gl;
            }
            __syncthreads();
        }
        const float delta = s_delta;
        float ub = -INFINITY;
        if (kn.ranking_fallback) {
            ubm = warp_max(sh.red_f[0][lane & (NW - 1)]);
            ub = __fadd_rn(ubm, delta);
        }
        if (warp == 0) {
            ct->top_blocks[lane] = lane < rk ? top_idx[lane] : -1;
            ct->fp16_scores[lane] = lane < rk ? top_f16[lane] : 0.0f;
            ct->fp16_logmass[lane] = lane < rk ? top_lm[lane] : 0.0f;
            // lane i owns candidate i (candidates are in INT8 order): its position in the stable
            // descending FP16 order, and in the descending FP16 log-mass order
            const bool mine = lane < rk;
            const float fs = mine ? top_f16[lane] : 0.0f;
            const float lmv = mine ? top_lm[lane] : 0.0f;
            int pos16 = 0, poslm = 0;
#pragma unroll 1
            for (int j = 0; j < rk; ++j) {
                const float fj = top_f16[j], lj = top_lm[j];
                pos16 += (fj > fs || (fj == fs && j < lane)) ? 1 : 0;
                poslm += (lj > lmv || (lj == lmv && j < lane)) ? 1 : 0;
            }
            const int r_main = min(kn.ranking_r, rk);
            const bool rf = kn.ranking_fallback && kn.ranking_r > 0;
            const bool d = mine && pos16 != lane;
            const int dis_main = (rf && __any_sync(FULL, d && lane < r_main)) ? 1 : 0;
            const int dis_r1 = (rf && __any_sync(FULL, d && lane < 1)) ? 1 : 0;
            const int dis_r3 = (rf && __any_sync(FULL, d && lane < 3)) ? 1 : 0;
            const unsigned who_r = __ballot_sync(FULL, mine && poslm == r_main - 1);
            const unsigned who_1 = __ballot_sync(FULL, mine && pos16 == 0);
            const unsigned who_2 = __ballot_sync(FULL, mine && pos16 == 1);
            float ell_r = -INFINITY;
            if (kn.ranking_fallback && r_main > 0) ell_r = __shfl_sync(FULL, lmv, __ffs(who_r) - 1);
            const float top1 = __shfl_sync(FULL, fs, __ffs(who_1) - 1);
            const float top2 = who_2 ? __shfl_sync(FULL, fs, __ffs(who_2) - 1) : top1;
            const int boundary = (kn.ranking_fallback && r_main > 0 && ub > ell_r) ? 1 : 0;
            int violation = 0;
            if (kn.score_consistency) {
                const float thr = __fadd_rn(delta, kn.eps_guard);
                violation = __any_sync(FULL, mine && fabsf(__fsub_rn(fs, top_i8[lane])) > thr) ? 1 : 0;
            }
            if (lane == 0) {
                const int rung3 = (dis_main | boundary) ? 1 : 0;
                ct->ranking_disagree = dis_main;
                ct->ranking_disagree_r1 = dis_r1;
                ct->ranking_disagree_r3 = dis_r3;
                ct->boundary_triggered = boundary;
                ct->rung3 = rung3;
                ct->consistency_violation = violation;
                ct->delta = delta;
                ct->boundary_ub = ub;
                ct->ell_fp16_r = ell_r;
                ct->fp16_top1 = top1;
                ct->fp16_top2 = top2;
                ct->int8_top1 = top_i8[0];
                const int dense = (kn.ranking_fallback && kn.rung3_recompute && rung3) ? 1 : 0;
                ct->dense = dense;
                if (dense) {
                    const int slot = atomicAdd(ws.any_flags + 4, 1);
                    if (slot < (int)gridDim.x) ws.any_flags[5 + slot] = h;
                }
                if (rung3) atomicOr(ws.any_flags + 1, 1);
                if (violation) atomicOr(ws.any_flags + 2, 1);
            }
        }
    } else if (role == 1 && tid == 0) {
        ct->ranking_disagree = ct->ranking_disagree_r1 = ct->ranking_disagree_r3 = 0;
        ct->boundary_triggered = ct->rung3 = ct->consistency_violation = ct->dense = 0;
        ct->delta = 0.0f;
        ct->boundary_ub = -INFINITY;
        ct->ell_fp16_r = -INFINITY;
        ct->fp16_top1 = ct->fp16_top2 = ct->int8_top1 = 0.0f;
        for (int i = 0; i < CQA_MAX_RANKING_K; ++i) { ct->top_blocks[i] = -1; ct->fp16_scores[i] = 0.0f; ct->fp16_logmass[i] = 0.0f; }
    }
    if (role == 1) return;

    // ---- Rung-2 value check (A holds the contributions mass fraction * eta_b, C still holds eta_b)
    unsigned char *vm = ws.value_mask + (long)h * ws.ld;
    if (!have_int4) {
        for (int b = tid; b < (int)nact; b += NT) vm[b] = 1;   // FP16-value cache: every block reads Tier 2
        if (tid == 0) { ct->e_pre = 0.0f; ct->e_val = 0.0f; ct->value_promoted_blocks = 0; }
        return;
    }
    const float *e = A;
    // Greedy promotion, largest contribution first (ties: lower block id first): block b is promoted while the
    // column sum of the contributions ranked before it is below the excess.  That sum never decreases along the
    // ranking, so the promoted blocks are exactly those with contribution bits >= t0, where t0 is the largest
    // threshold whose admitted set still sums to at least the excess (no sort, no serial walk).  Exact ties at t0
    // are resolved the same way over the block id.
    int cnt = 0;
    const float e_pre = column_sum1<NT>(e, n, sh, parity, cnt, [](unsigned, int) { return true; });
    const float excess = fmaxf(__fsub_rn(e_pre, kn.v_tolerance), 0.0f);
    float promoted = 0.0f;
    int n_prom = 0;
    unsigned t0 = 0xFFFFFFFFu;   // nothing admitted
    int id_bound = 0;
    if (kn.value_mode_tight) {
        if (excess > 0.0f) {
            t0 = 0u;
            int cnt_lo = cnt, cnt_hi = 0;     // entries >= t0, entries >= the upper end of the open range
            float f_lo = e_pre, f_hi = 0.0f;  // their column sums
            int bit = 30;
            // Hints first: bins over the top 11 bits of the contributions (then over the next 11 of the bin found, then
            // over the last 9), each holding a fixed-point sum of its entries (integer atomics; the scale keeps the
            // total below 2^30).  The bin where the approximate suffix sum crosses the excess is then CHECKED with
            // exact column sums of its two edges (and of a neighbour's, if it is one bin off); only if the exact sums
            // bracket the excess does the search continue inside the bin.  Where they do not it goes on bit by bit from
            // what is certain.  The result never depends on the approximation.  (Diffuse attention leaves hundreds of
            // entries in the first bin: ten passes over the blocks for its 20 open bits, three with a second hint.)
            float emax = 0.0f;
            if (n > 64) {
#pragma unroll 1
                for (int k = 0; k < nk; ++k) {
                    const int b = k * NT + tid;
                    if (b < n) emax = fmaxf(emax, e[b]);
                }
                emax = cta_max<NT>(emax, sh, parity);
            }
            int *hsum = reinterpret_cast<int *>(B);
#pragma unroll 1
            for (int level = 0; level < 3 && emax > 0.0f && cnt_lo - cnt_hi > (level == 0 ? 1 : 3); ++level) {
                const int shift = level == 0 ? 20 : (level == 1 ? 9 : 0), nbins = level == 2 ? 512 : 2048;
                // entries of the open range [t0, t_end), their number and an upper bound of them
                const unsigned t_end = level == 0 ? 0x80000000u : t0 + (1u << (level == 1 ? 20 : 9));
                const float vmax = level == 0 ? emax : __uint_as_float(t_end);
                const int members = cnt_lo - cnt_hi;
                hist_clear<NT>(hsum);
                __syncthreads();
                const float sc = __fdiv_rn(1073741824.0f, __fmul_rn((float)members, vmax));     // 2^30 / (members * max)
#pragma unroll 1
                for (int k = 0; k < nk; ++k) {
                    const int b = k * NT + tid;
                    const float v = b < n ? e[b] : 0.0f;
                    const unsigned x = __float_as_uint(v);
                    const int qv = (int)__fmul_rn(v, sc);
                    hist_add(hsum, x >= t0 && x < t_end && qv > 0, (x >> shift) & (unsigned)(nbins - 1), qv);
                }
                __syncthreads();
                const int need = max(1, (int)fminf(__fmul_rn(fmaxf(__fsub_rn(excess, f_hi), 0.0f), sc), 1073741824.0f));
                int above, in_bin;
                const int d = find_suffix_crossing<NT>(hsum, nbins, need, sh, above, in_bin);
                if (d < 0) break;
                const unsigned one = 1u << shift, t_lo = t0 + ((unsigned)d << shift), t_hi = t_lo + one;
                float fs[3];
                int cs3[3];
                column_sums3<NT>(e, n, t_lo, t_hi, 0xFFFFFFFFu, sh, parity, fs, cs3);
                bool found = true;
                if (fs[0] >= excess && fs[1] < excess) {
                    t0 = t_lo; cnt_lo = cs3[0]; f_lo = fs[0]; cnt_hi = cs3[1]; f_hi = fs[1];
                } else {
                    // the fixed-point sums put the crossing one bin off: look at the neighbour on that side
                    const unsigned t_dn = d > 0 ? t_lo - one : t0;
                    const unsigned t_up = d + 2 < nbins ? t_hi + one : 0xFFFFFFFFu;
                    float gs[3];
                    int gc[3];
                    column_sums3<NT>(e, n, t_dn, t_up, 0xFFFFFFFFu, sh, parity, gs, gc);
                    if (d > 0 && fs[0] < excess && gs[0] >= excess) {
                        t0 = t_dn; cnt_lo = gc[0]; f_lo = gs[0]; cnt_hi = cs3[0]; f_hi = fs[0];
                    } else if (d + 2 < nbins && fs[1] >= excess && gs[1] < excess) {
                        t0 = t_hi; cnt_lo = cs3[1]; f_lo = fs[1]; cnt_hi = gc[1]; f_hi = gs[1];
                    } else {
                        found = false;
                    }
                }
                if (!found) break;
                bit = shift - 1;
                __syncthreads();         // the bins are cleared again
            }
            // two bits per step: of the three trial thresholds t0 + {1,2,3} << (bit-1), keep the highest whose admitted
            // entries still reach the excess (the sums fall as the threshold rises)
#pragma unroll 1
            for (; bit >= 1 && cnt_lo - cnt_hi > 1; bit -= 2) {
                const unsigned s1 = t0 | (1u << (bit - 1)), s2 = t0 | (2u << (bit - 1)), s3 = t0 | (3u << (bit - 1));
                float fs[3];
                int cs3[3];
                column_sums3<NT>(e, n, s1, s2, s3, sh, parity, fs, cs3);
                if (fs[2] >= excess) { t0 = s3; cnt_lo = cs3[2]; f_lo = fs[2]; }
                else if (fs[1] >= excess) { t0 = s2; cnt_lo = cs3[1]; f_lo = fs[1]; cnt_hi = cs3[2]; }
                else if (fs[0] >= excess) { t0 = s1; cnt_lo = cs3[0]; f_lo = fs[0]; cnt_hi = cs3[1]; }
                else cnt_hi = cs3[0];
            }
            if (bit == 0 && cnt_lo - cnt_hi > 1) {      // an odd number of bits was open (search from the top: 31)
                const unsigned trial = t0 | 1u;
                int cc = 0;
                const float fv = column_sum1<NT>(e, n, sh, parity, cc, [=](unsigned x, int) { return x >= trial; });
                if (fv >= excess) { t0 = trial; cnt_lo = cc; f_lo = fv; } else { cnt_hi = cc; }
            }
            promoted = f_lo;
            n_prom = cnt_lo;
            id_bound = n;                     // every entry equal to t0 is admitted ...
            if (cnt_lo - cnt_hi > 1) {
                // ... unless several entries equal t0: admit them in block order while the sum stays below
                int i0 = 0;
#pragma unroll 1
                for (int bit2 = 14; bit2 >= 0; --bit2) {
                    const int trial = i0 | (1 << bit2);
                    if (trial > n) continue;
                    int cc = 0;
                    const float g = column_sum1<NT>(e, n, sh, parity, cc, [=](unsigned x, int b) { return x > t0 || (x == t0 && b < trial); });
                    if (g < excess) i0 = trial;
                }
                id_bound = i0 + 1;
                const int bound = id_bound;
                promoted = column_sum1<NT>(e, n, sh, parity, n_prom, [=](unsigned x, int b) { return x > t0 || (x == t0 && b < bound); });
            }
        }
    } else {
        // loose mode: every block whose eta_b exceeds the tolerance
        const float vt = kn.v_tolerance;
        promoted = column_sum1<NT>(e, n, sh, parity, n_prom, [=](unsigned, int b) { return C[b] > vt; });
    }
#pragma unroll 1
    for (int k = 0; k < nk; ++k) {
        const int b = k * NT + tid;
        if (b < n) {
            unsigned char upb;
            if (kn.value_mode_tight) {
                const unsigned bits = __float_as_uint(e[b]);
                upb = (t0 != 0xFFFFFFFFu && (bits > t0 || (bits == t0 && b < id_bound))) ? 1 : 0;
            } else {
                upb = C[b] > kn.v_tolerance ? 1 : 0;
            }
            vm[b] = upb;
        }
    }
    // the trailing partial block (at most one) lies beyond the blocks the threads own
    if (tid == 0 && (int)nact > n) vm[n] = kn.force_trailing_value_fp16 ? 1 : 0;
    if (tid == 0) {
        ct->e_pre = e_pre;
        ct->e_val = fmaxf(__fsub_rn(e_pre, promoted), 0.0f);
        ct->value_promoted_blocks = n_prom;
        if (n_prom > 0) atomicOr(ws.any_flags + 3, 1);
    }
}

template <int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) selcert_kernel(const __grid_constant__ cqa_cache c, const __grid_constant__ cqa_knobs kn,
                                                                const __grid_constant__ cqa_workspace ws, const void *q,
                                                                int q_dtype, long nq, long nact, const float *u, long u_ld,
                                                                int n_pad, int hi, int base_width, int two_level, int rk,
                                                                int phases, int role_base)
{
    selcert_body<NT>(c, kn, ws, q, q_dtype, nq, nact, u, u_ld, n_pad, hi, base_width, two_level, rk, phases, role_base);
}

static __host__ __device__ inline int next_pow2(long n)
{
    int p = 32;
    while (p < n) p <<= 1;
    return p;
}

// Selection widths derived from the knobs (shared by the argument check, the launch and the batched kernel).
struct SelPlan {
    int hi, base_width, two_level, rk;
};
static __host__ __device__ inline SelPlan sel_plan(const cqa_knobs *kn, long nq)
{
    SelPlan p;
    const bool can_expand = kn->rung1_threshold >= 0.0f && kn->k_max > 0;
    long sel_kmax = kn->k_max;
    p.two_level = 0;
    if (can_expand) {
        long expanded = (long)ceil((double)kn->k_max * (double)kn->rung1_multiplier);
        if (expanded > nq) expanded = nq;
        if (expanded > kn->k_max) { sel_kmax = expanded; p.two_level = 1; }
    }
    p.hi = (int)(sel_kmax <= 0 ? nq : (sel_kmax < nq ? sel_kmax : nq));
    p.base_width = p.two_level ? (int)(kn->k_max < p.hi ? kn->k_max : p.hi) : p.hi;
    int rk = kn->ranking_r > kn->top_k_fp16_keys ? kn->ranking_r : kn->top_k_fp16_keys;
    if (rk < 4) rk = 4;
    if (rk > nq) rk = (int)nq;
    p.rk = rk;
    return p;
}

// Sequence blockIdx.z of a batch: the fused selector + certifier (all three roles) with that sequence's sizes.
template <int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) selcert_batched_kernel(const cqa_batch_item *items, cqa_knobs kn, int q_dtype,
                                                                        int do_append)
{
    const cqa_batch_item &it = *stage_batch_item(items + blockIdx.z);
    const long num_tokens = it.pos + do_append;
    const long nq = num_tokens / BS, nact = (num_tokens + BS - 1) / BS;
    const SelPlan p = sel_plan(&kn, nq);
    selcert_body<NT>(it.cache, kn, it.ws, it.q, q_dtype, nq, nact, nullptr, 0, next_pow2(nq), p.hi, p.base_width, p.two_level,
                      p.rk, PH_SELECT | PH_CERTIFY | PH_FLAGS_CLEARED, 0);
}

static size_t selcert_smem(int n_pad)
{
    const size_t n_arr = n_pad > 2048 ? n_pad : 2048;
    return n_arr * 8 + (size_t)n_pad * 5 + (size_t)LIST * 8 + (size_t)CAND * 4 + ((size_t)((n_pad > 1024 ? n_pad : 1024) >> 5) + (n_pad >> 8) + 8) * 4 + 64;
}

// Every argument check of the selector / certifier launch; nothing is launched or copied here.
int selcert_check(const cqa_cache *c, const cqa_knobs *kn, const cqa_workspace *ws, const void *q, long nq, int phases)
{
    if (nq <= 0) { set_error("selector: needs at least one quantised block"); return CQA_ERR_INVALID; }
    if (nq > CQA_MAX_SORT_BLOCKS) {
        set_error("selector: %ld quantised blocks exceed the limit %d", nq, CQA_MAX_SORT_BLOCKS);
        return CQA_ERR_TOO_LARGE;
    }
    if (nq > ws->ld && ws->shard_stride <= 0) { set_error("selector: workspace ld %ld < %ld blocks", (long)ws->ld, nq); return CQA_ERR_INVALID; }
    if (c->t2_dtype < 0 || c->t2_dtype > 2) { set_error("selector: unknown Tier-2 dtype %d", c->t2_dtype); return CQA_ERR_INVALID; }
    const SelPlan p = sel_plan(kn, nq);
    if ((phases & PH_SELECT) && ws->sel_width < p.hi) {
        set_error("cqa_select: workspace sel_width %d < required %d", ws->sel_width, p.hi);
        return CQA_ERR_INVALID;
    }
    if (p.rk > CQA_MAX_RANKING_K - 1) {
        set_error("cqa_certify: ranking set of %d blocks exceeds the limit %d", p.rk, CQA_MAX_RANKING_K - 1);
        return CQA_ERR_TOO_LARGE;
    }
    if (phases & PH_CERTIFY) {
        const bool need_fp16 = kn->ranking_fallback || kn->score_consistency;
        const bool local_keys = !(phases & (PH_TOP_ONLY | PH_GIVEN));
        if ((phases & PH_PEER_B) && (ws->peer_world < 2 || ws->peer_world > 8 || !ws->given_fp16 || ws->peer_step < 1)) {
            set_error("selector: incomplete peer description for the in-kernel exchange");
            return CQA_ERR_INVALID;
        }
        if (need_fp16 && c->sigma_max && ((uintptr_t)c->sigma_max & 15)) {
            set_error("cqa_certify: sigma_max must be 16-byte aligned");
            return CQA_ERR_INVALID;
        }
        if (need_fp16 && local_keys && (!c->keys_t2 || !c->sigma_max || !q)) {
            set_error("cqa_certify: ranking / consistency checks need q, Tier-2 keys and sigma_max");
            return CQA_ERR_INVALID;
        }
        if (need_fp16 && (phases & PH_GIVEN) && (!ws->given_fp16 || !c->sigma_max || !q)) {
            set_error("cqa_certify_given: needs q, sigma_max and the exchanged FP16 scores");
            return CQA_ERR_INVALID;
        }
    }
    return CQA_OK;
}

// Threads of a selector CTA for `nq` blocks and `ctas` CTAs.  A CTA takes about 5 + nq / NT units of 3.2 K cycles (a fixed
// chain of barriers and reductions, and one round per NT blocks) and 1024 / NT of them fit an SM, so one sequence, whose
// CTAs have an SM each, wants many threads and a batch of short ones few: 32 sequences of 8192 tokens 443 us a step
// with 1024 threads, 353 with 512, 319 with 256; four of 65536 tokens 425 / 417 / 432; one of 32768 66 / 68 / 75.
static int selcert_threads(long nq, long ctas)
{
    int best = 1024;
    double best_cost = 0.0;
    for (int nt = 1024; nt >= 256; nt /= 2) {
        const double slots = (double)sm_count() * (1024 / nt);
        const double cost = (ctas > slots ? ctas / slots : 1.0) * (5.0 + (double)nq / nt);
        if (nt == 1024 || cost < best_cost) { best = nt; best_cost = cost; }
    }
    return best;
}

template <int NT>
static int selcert_launch_v(const cqa_cache *c, const cqa_knobs *kn, const cqa_workspace *ws, const void *q,
                            int q_dtype, long nq, long nact, const float *u, long u_ld, int phases, int n_pad,
                            cudaStream_t st)
{
    const int H = c->kv_heads * c->gqa_group;
    const SelPlan p = sel_plan(kn, nq);
    const size_t smem = selcert_smem(n_pad);
    static size_t granted[SMEM_ATTR_DEVICES] = {};
    const int rc_attr = check_cuda(ensure_dynamic_smem(selcert_kernel<NT>, smem, granted), "cudaFuncSetAttribute(selcert_kernel)");
    if (rc_attr) return rc_attr;
    if ((phases & PH_SELECT) && !(phases & PH_FLAGS_CLEARED)) {
        int rc = check_cuda(cudaMemsetAsync(ws->any_flags, 0, (5 + H) * sizeof(int32_t), st),
                            "cudaMemsetAsync(any_flags)");
        if (rc) return rc;
    }
    // select only: role 0; certify only: roles 1 and 2; fused: all three
    const int role_base = (phases & PH_SELECT) ? 0 : 1;
    int n_roles = (phases & PH_SELECT) ? ((phases & PH_CERTIFY) ? 3 : 1) : 2;
    if (phases & PH_GIVEN) n_roles = 1;   // role 1 alone
    dim3 grid((unsigned)H, (unsigned)n_roles);
    // chained to the score kernel only in the fused step (a memset precedes the launch otherwise)
    const bool chained = (phases & PH_FLAGS_CLEARED) != 0;
    return check_cuda(launch_chained(selcert_kernel<NT>, grid, dim3(NT), smem, st, chained, *c, *kn, *ws, q, q_dtype,
                                     nq, nact, u, u_ld, n_pad, p.hi, p.base_width, p.two_level, p.rk, phases, role_base),
                      "selcert_kernel");
}

int selcert_launch(const cqa_cache *c, const cqa_knobs *kn, const cqa_workspace *ws, const void *q, int q_dtype,
                   long nq, long nact, const float *u, long u_ld, int phases, cudaStream_t st)
{
    const int rc = selcert_check(c, kn, ws, q, nq, phases);
    if (rc) return rc;
    const int n_pad = next_pow2(nq);
    switch (selcert_threads(nq, (long)c->kv_heads * c->gqa_group * 3)) {
    case 256: return selcert_launch_v<256>(c, kn, ws, q, q_dtype, nq, nact, u, u_ld, phases, n_pad, st);
    case 512: return selcert_launch_v<512>(c, kn, ws, q, q_dtype, nq, nact, u, u_ld, phases, n_pad, st);
    default: return selcert_launch_v<1024>(c, kn, ws, q, q_dtype, nq, nact, u, u_ld, phases, n_pad, st);
    }
}

template <int NT>
static int selcert_batched_launch_v(const cqa_batch_item *items_dev, int n_items, int n_heads, int n_pad, const cqa_knobs *kn,
                                    int q_dtype, int do_append, cudaStream_t st)
{
    const size_t smem = selcert_smem(n_pad);
    dim3 grid((unsigned)n_heads, 3u, (unsigned)n_items);
    static size_t granted[SMEM_ATTR_DEVICES] = {};
    const int rc = check_cuda(ensure_dynamic_smem(selcert_batched_kernel<NT>, smem, granted),
                              "cudaFuncSetAttribute(selcert_batched_kernel)");
    if (rc) return rc;
    return check_cuda(launch_chained(selcert_batched_kernel<NT>, grid, dim3(NT), smem, st, true, items_dev, *kn, q_dtype,
                                     do_append), "selcert_batched_kernel");
}

// The selector of a batch; `max_nq` = most quantised blocks of any sequence (sizes the shared memory), every item checked by the caller.
int selcert_batched_launch(const cqa_batch_item *items_dev, int n_items, int n_heads, long max_nq, const cqa_knobs *kn,
                           int q_dtype, int do_append, cudaStream_t st)
{
    const int n_pad = next_pow2(max_nq);
    switch (selcert_threads(max_nq, (long)n_heads * 3 * n_items)) {
    case 256: return selcert_batched_launch_v<256>(items_dev, n_items, n_heads, n_pad, kn, q_dtype, do_append, st);
    case 512: return selcert_batched_launch_v<512>(items_dev, n_items, n_heads, n_pad, kn, q_dtype, do_append, st);
    default: return selcert_batched_launch_v<1024>(items_dev, n_items, n_heads, n_pad, kn, q_dtype, do_append, st);
    }
}

int selcert_wait_timeouts(int *count, int reset) { return wait_timeouts_of_this_unit(count, reset); }

int select_launch(const cqa_cache *c, const cqa_knobs *kn, const cqa_workspace *ws, long nq, long nact,
                  const float *u, long u_ld, cudaStream_t st)
{
    return selcert_launch(c, kn, ws, nullptr, CQA_F32, nq, nact, u, u_ld, PH_SELECT, st);
}

int select_certify_local_launch(const cqa_cache *c, const cqa_knobs *kn, const cqa_workspace *ws, long nq,
                                long nact, const float *u, long u_ld, cudaStream_t st)
{
    return selcert_launch(c, kn, ws, nullptr, CQA_F32, nq, nact, u, u_ld, PH_SELECT | PH_CERTIFY | PH_TOP_ONLY, st);
}

int certify_given_launch(const cqa_cache *c, const cqa_knobs *kn, const cqa_workspace *ws, const void *q,
                         int q_dtype, long nq, long nact, cudaStream_t st)
{
    return selcert_launch(c, kn, ws, q, q_dtype, nq, nact, nullptr, 0, PH_CERTIFY | PH_GIVEN, st);
}

int certify_launch(const cqa_cache *c, const cqa_knobs *kn, const cqa_workspace *ws, const void *q, int q_dtype,
                   long nq, long nact, cudaStream_t st)
{
    return selcert_launch(c, kn, ws, q, q_dtype, nq, nact, nullptr, 0, PH_CERTIFY, st);
}

}  // namespace cqa
