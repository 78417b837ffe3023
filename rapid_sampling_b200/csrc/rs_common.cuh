// Pieces shared by the sampler kernels: launch parameters, the per-row argument record, the strided row view
// used by the whole-row search, and the element-wise arithmetic (scaled / penalised logits) that every variant
// must compute with the same operations in the same order.  sm_100a only.
#pragma once
#include "rs_device.cuh"
#include "../../include/rapid_sampling_b200.h"

namespace rs {

enum Kind : int { kTopP = 0, kGeneral = 1, kRepetition = 2 };

struct Params {
    const void* logits;      // already offset to position T-1 of row 0; fp32, fp16 or bf16 (dtype)
    int dtype;               // RS_DTYPE_F32 / F16 / BF16 of the logits
    long long row_stride;    // elements between consecutive rows (T*V)
    float* penalties;        // (B,V) or null
    unsigned char* states;   // B*64
    int* out;                // B
    float* scratch;          // B*V floats (global-row variant only)
    float* dbg_probs;        // optional (B,V)
    rs_trace* dbg_trace;     // optional B
    int* status;             // device status word
    int* status_mirror;      // optional: a word of pinned host memory the device can write (zero-copy), or null
    uint32_t wait_polls;     // polls after which a bounded wait gives up
    int B, V, kind, top_k;
    int sel_rank;            // 0 = no candidate shortcut; else rank of the per-warp thread maximum used as bound
    int cand_slots;          // float4 slots per lane of the candidate buffer (shared-memory variant)
    float scale, top_p, presence, repetition, decay;
    const struct RowArgs* rows;   // per-row parameters (ROWP kernels only), else null
    const int* route;        // per-row parameters: word the rows' settings decide (1: some row searches widely), or null
    int route_is;            // the kernel runs only if the word holds this
    float* out_prob;         // optional B: probability of the sampled id (ROWP kernels only)
    float* out_kept;         // optional B: kept probability mass the id was drawn from (ROWP kernels only)
    int quick;               // 1: try the search on integer masses first; 0 (test instrumentation): exact search only
};

// Normalised parameters of one row, made on the device from the caller's per-row tensors.
struct __align__(32) RowArgs {
    int kind, top_k, sel_rank, pad0;
    float scale, top_p, pad1, pad2;
};

// shared-memory map (bytes)
constexpr int kXWords = 10;                      // words each warp contributes to an exchange
template <int N> struct Packets { static constexpr int value = N; };   // 16-byte packets of an exchange record
constexpr int kXStride = 12;                     // words between two warps' records in a mailbox (16-byte aligned records)
constexpr int kMboxOff = 0;                      // 2 buffers of [32 warps][kXStride] words
constexpr int kMboxBuf = kXStride * 32 * 4;
constexpr int kMiscOff = 2 * kMboxBuf;           // mbarriers, small scalars, 32 warp totals
constexpr int kQuickCap = 512;                   // longest candidate list the search on integer masses takes
constexpr int kQsumOff = kMiscOff + 256;         // counts and masses at that search's 32 samples
constexpr int kQuickOff = kQsumOff + 256;        // the row's candidates as one unordered list of (bits of p, p in units of 2^-30)
constexpr int kSlabOff = kQuickOff + kQuickCap * 8;
constexpr uint32_t kDefaultWaitPolls = 1u << 22;

__host__ __device__ constexpr int slab_bytes(int V, int C) { return ((V / 4 + 1023) / 1024) * (1024 / C) * 16; }

template <int C, bool SMEM>
struct Row {
    static constexpr int L = kLanes / C;
    float4* slab;
    int t, tg;
    __device__ __forceinline__ float4 ld(int s) const { return SMEM ? slab[s * L + t] : slab[s * kLanes + tg]; }
    __device__ __forceinline__ void st(int s, float4 v) const {
        if (SMEM) slab[s * L + t] = v; else slab[s * kLanes + tg] = v;
    }
};

// Probability of one element, exactly as the streaming passes compute it.
__device__ __forceinline__ float scaled_logit(float l, float pen, bool rep, float scale) {
    return rep ? sanitize((sanitize(l) - pen) * scale) : sanitize(l * scale);
}

// One search pass over this lane's list in the slab: ordered masses and counts at three pivots
// (f[3] is ignored here); optionally keeps only elements >= keepf (in place, order preserved, tail
// padded with -1).  Counts are returned packed: c01 = n(f0) | n(f1) << 16, c23 = n(f2).
template <int C, bool SMEM, bool COMPACT>
__device__ __forceinline__ void slab_pass(const Row<C, SMEM>& row, int& n, const float (&f)[4], float keepf, float (&m)[4],
                                          uint32_t& c01, uint32_t& c23) {
    uint32_t cy = 0, cz = 0, cw = 0;
    float my = 0.f, mz = 0.f, mw = 0.f;
    const float py = f[0], pz = f[1], pw = f[2];
    const int slots = (n + 3) >> 2;
    float b0 = -1.f, b1 = -1.f, b2 = -1.f, b3 = -1.f;
    int q = 0;
#pragma unroll ((SMEM || COMPACT || C > 1) ? 2 : 4)
    for (int s = 0; s < slots; s++) {
        const float4 v = row.ld(s);
        const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float p = e[j];
            if (p >= py) { cy++; my += p; }
            if (p >= pz) { cz++; mz += p; }
            if (p >= pw) { cw++; mw += p; }
            if (COMPACT) {
                if (p >= keepf) {
                    const int k = q & 3;
                    b0 = (k == 0) ? p : b0;
                    b1 = (k == 1) ? p : b1;
                    b2 = (k == 2) ? p : b2;
                    b3 = (k == 3) ? p : b3;
                    q++;
                    if ((q & 3) == 0) {
                        row.st((q >> 2) - 1, make_float4(b0, b1, b2, b3));
                        b0 = b1 = b2 = b3 = -1.f;
                    }
                }
            }
        }
    }
    if (COMPACT) {
        if (q & 3) row.st(q >> 2, make_float4(b0, b1, b2, b3));
        n = q;
    }
    m[0] = my; m[1] = mz; m[2] = mw; m[3] = 0.f;
    c01 = cy | (cz << 16);
    c23 = cw;
}

// ---- the cutoff search of a whole row's candidate list, on integer masses ---------------------------------------
// The reference's loop only ever asks whether a mass is below or above top_p (sampling.cu:598, :618-651).  `list`
// holds every candidate of the row as (bits of p, p in units of 2^-30), in any order: the sum of the admitted
// entries' second words is exact up to half a unit per entry and does not depend on the order.  The reference's fp32
// value differs from the true sum by at most one rounding per addition on the longest path (`depth`: the entries of
// one lane, 5 in the warp tree, 31 over the warps).  Outside that margin around top_p the answer is certain; inside it
// (unless a count decides the test anyway) the verdict is 0 and the caller runs the exact search from the start.
// Pivots at or below beta_p are answered by the set {p > beta_p}, as in the exact search on a candidate list.
//
// The answer at a pivot u depends only on the set {p >= u}, which shrinks as u rises: every entry up to some x2 has a
// set that exceeds top_k or top_p, every entry above some x has one that passes, and between the two lie those where
// neither is certain.  So x2 and x are found first and the loop is then replayed -- same pivots, same tests, same
// bracket updates -- on two integer compares per test, without reading the list.  x2 and x are found by rank: 32
// entries of the list as sample, each lane sums the sets of one of them (quick_sample: the list is split over the warps
// of the CTA), which leaves about a thirty-second of the list between the highest sample that exceeds and the lowest
// that passes; one warp ranks those against each other (quick_settle).  Bound by the latency of one warp: replaying the
// loop with a scan of the list in each of its ~14 rounds took 2 us longer (a call of B=1, V=262144: 20.0 -> 18.2 us).
struct QuickTest {       // the three possible outcomes of the reference's tests at a set of count c and mass m
    bool use_cnt;
    uint32_t top_k, tp_lo, tp_hi, margin;
    // depth: additions on the longest path of the reference's sum; cap: longest list (half a unit of rounding per entry)
    __device__ __forceinline__ QuickTest(bool uc, uint32_t k, float top_p, int depth, int cap = kQuickCap) {
        use_cnt = uc;
        top_k = k;
        margin = (uint32_t)(depth * 66 + cap / 2 + 8);
        tp_lo = __float2uint_rd(top_p * 1073741824.f);
        tp_hi = __float2uint_ru(top_p * 1073741824.f);
    }
    // 2: more than top_k entries or more than top_p mass for certain; 0: fewer and less for certain; 1: neither test
    // (count equal to top_k); 3: the mass is too close to top_p to tell
    __device__ __forceinline__ int operator()(uint32_t c, uint32_t m) const {
        const bool lt = m + margin < tp_lo, gt = m > tp_hi + margin, many = use_cnt && c > top_k;
        if (gt || many) return 2;
        if (!lt) return 3;
        return (!use_cnt || c < top_k) ? 0 : 1;
    }
};

// First part, all NW warps of the CTA: counts and masses at the 32 samples into sums[0..31], sums[32..63] (cleared by
// the caller; complete after the next CTA barrier).
template <int NW>
__device__ __forceinline__ void quick_sample(const uint2* list, const uint32_t n, const int w, const int lane, uint32_t* sums) {
    const uint32_t pv = list[((uint32_t)lane * n) >> 5].x;
    const uint32_t chunk = (n + NW - 1) / NW, i0 = (uint32_t)w * chunk, i1 = min(n, i0 + chunk);
    uint32_t c = 0u, m = 0u;
#pragma unroll 8
    for (uint32_t i = i0; i < i1; i++) {
        const uint2 e = list[i];
        if (e.x >= pv) { c++; m += e.y; }
    }
    atomicAdd(sums + lane, c);
    atomicAdd(sums + 32 + lane, m);
}

// Second part, one warp (all 32 lanes, same arguments).  The list is compacted in place.
// Verdict: 1 settled (left / right / rounds are the reference's), 2 the list cannot settle the cutoff, 0 undecided.
__device__ __forceinline__ int quick_settle(uint2* list, const uint32_t n, const int lane, const uint32_t* sums, const QuickTest test,
                                            const float top_p, const uint32_t beta_p, const float pmin, const float pmax,
                                            const uint32_t V, uint32_t& left, uint32_t& right, uint32_t& rounds) {
    constexpr unsigned FULLW = 0xffffffffu;
    uint32_t x2 = 0u;                                    // every entry up to here exceeds
    uint32_t x0 = 0xffffffffu, base_c = 0u, base_m = 0u; // every entry from here on passes; count and mass of that set
    uint32_t nz = n, pv = list[((uint32_t)lane * n) >> 5].x, c = sums[lane], m = sums[32 + lane];
    for (int it = 0;; it++) {
        const int cls = test(c, m);
        x2 = max(x2, __reduce_max_sync(FULLW, cls == 2 ? pv : 0u));
        const uint32_t low = __reduce_min_sync(FULLW, cls == 0 ? pv : 0xffffffffu);
        if (low < x0) {
            const int src = __ffs(__ballot_sync(FULLW, cls == 0 && pv == low)) - 1;
            x0 = low;
            base_c = __shfl_sync(FULLW, c, src);
            base_m = __shfl_sync(FULLW, m, src);
        }
        // what lies between: compacted to the front of the list (a place is written only after it has been read)
        const uint32_t lo = max(x2, beta_p);
        uint32_t q = 0u;
        for (uint32_t i0 = 0u; i0 < nz; i0 += 128u) {
            uint2 e[4];
            unsigned b[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const uint32_t i = i0 + (uint32_t)(32 * j + lane);
                e[j] = (i < nz) ? list[i] : make_uint2(0u, 0u);
            }
#pragma unroll
            for (int j = 0; j < 4; j++) b[j] = __ballot_sync(FULLW, e[j].x > lo && e[j].x < x0);
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if ((b[j] >> lane) & 1u) list[q + (uint32_t)__popc(b[j] & ((1u << lane) - 1u))] = e[j];
                q += (uint32_t)__popc(b[j]);
            }
            __syncwarp();
        }
        __syncwarp();
        nz = q;
        if (nz <= 32u || it == 3) break;
        pv = list[((uint32_t)lane * nz) >> 5].x;
        c = base_c;
        m = base_m;
#pragma unroll 8
        for (uint32_t i = 0u; i < nz; i++) {
            const uint2 e = list[i];
            if (e.x >= pv) { c++; m += e.y; }
        }
    }
    uint32_t x = x2;
    bool unsure = false;
    for (uint32_t i0 = 0u; i0 < nz; i0 += 32u) {         // one turn (more only for masses of ties that cannot be told apart)
        const bool mine = i0 + (uint32_t)lane < nz;
        pv = mine ? list[i0 + (uint32_t)lane].x : 0xffffffffu;
        c = base_c;
        m = base_m;
#pragma unroll 4
        for (uint32_t i = 0u; i < nz; i++) {
            const uint2 e = list[i];
            if (e.x >= pv) { c++; m += e.y; }
        }
        const int cls = mine ? test(c, m) : 0;
        x2 = max(x2, __reduce_max_sync(FULLW, cls == 2 ? pv : 0u));
        x = max(x, __reduce_max_sync(FULLW, cls != 0 ? pv : 0u));
        unsure = unsure || __any_sync(FULLW, cls == 3);
    }
    x = max(x, x2);
    if (test(0u, 0u) != 0) { x = 0xffffffffu; unsure = true; }      // not even the empty set is clear of top_p

    const uint32_t ustar = beta_p + 1u;
    uint32_t l_left = __float_as_uint(pmin), l_right = __float_as_uint(pmax) + 1u, l_rounds = 0u;
    // whether the set at `left` keeps the loop going (the reference starts from the whole row and mass 1)
    bool go = (test.use_cnt && V > test.top_k) || 1.0f > top_p;
    int verdict = 1;
    while (go && l_left < l_right - 1u && l_rounds < 64u) {
        l_rounds++;
        const uint32_t pz = (l_left + l_right) >> 1, py = (l_left + pz) >> 1, pwv = (pz + l_right) >> 1;
        const uint32_t e0 = max(py, ustar), e1 = max(pz, ustar), e2 = max(pwv, ustar);
        const bool g0 = e0 <= x2, g1 = e1 <= x2, g2 = e2 <= x2;     // exceeds
        const bool s0 = e0 > x && py > beta_p, s1 = e1 > x && pz > beta_p, s2 = e2 > x && pwv > beta_p;   // passes
        if (unsure && ((!g0 && e0 <= x) || (!g1 && e1 <= x) || (!g2 && e2 <= x))) { verdict = 0; break; }
        if ((py <= beta_p && !g0) || (pz <= beta_p && !g1) || (pwv <= beta_p && !g2)) { verdict = 2; break; }
        const uint32_t nl = s0 ? l_left : s1 ? py : s2 ? pz : pwv;
        l_right = s0 ? py : s1 ? pz : s2 ? pwv : l_right;
        l_left = nl;
        go = s0 ? go : s1 ? g0 : s2 ? g1 : g2;
    }
    if (verdict == 1 && !(l_left > beta_p)) verdict = 2;
    left = l_left; right = l_right; rounds = l_rounds;
    return verdict;
}

// Sanitised scaled logit with the common case (finite product) kept to a multiply and a compare.
__device__ __forceinline__ float scaled_fast(float l, float scale) {
    const float x = l * scale;
    return (fabsf(x) <= FLT_MAX) ? x : sanitize(x);
}
// The rare path, kept out of line so that the streaming loops stay short.
__device__ __forceinline__ float4 sanitize4(float4 v) {
    return make_float4(sanitize(v.x), sanitize(v.y), sanitize(v.z), sanitize(v.w));
}
// Four scaled logits; a single test per group finds any Inf / NaN product (x * 0 is NaN exactly for those).
__device__ __forceinline__ float4 scaled4(float4 l, float scale) {
    float4 v = make_float4(l.x * scale, l.y * scale, l.z * scale, l.w * scale);
    const float probe = fmaf(v.w, 0.f, fmaf(v.z, 0.f, fmaf(v.y, 0.f, v.x * 0.f)));
    if (probe != probe) v = sanitize4(v);
    return v;
}
// Four penalised scaled logits, sanitize((sanitize(l) - pen) * scale).  If the plain product is finite, the logit
// was finite too (an Inf / NaN logit keeps the product non-finite for any finite or non-finite penalty), both
// sanitisers were identities and the product is the result; anything else takes the exact formula.
__device__ __forceinline__ float4 scaled4_rep(float4 l, float4 q, float scale) {
    float4 v = make_float4((l.x - q.x) * scale, (l.y - q.y) * scale, (l.z - q.z) * scale, (l.w - q.w) * scale);
    const float probe = fmaf(v.w, 0.f, fmaf(v.z, 0.f, fmaf(v.y, 0.f, v.x * 0.f)));
    if (probe != probe)
        v = make_float4(scaled_logit(l.x, q.x, true, scale), scaled_logit(l.y, q.y, true, scale),
                        scaled_logit(l.z, q.z, true, scale), scaled_logit(l.w, q.w, true, scale));
    return v;
}
// Correctly rounded quotients by one denominator (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34(1), 1990): y is the correctly rounded 1/b; the first correction makes q a
// neighbour of a/b (what it rounds is within 1.5 ulp * 2^-24 of a/b), and for such a q with an exact remainder the second
// one yields the rounded quotient.  Remainders are exact and nothing underflows for a >= kDivMin = 2^-78 (they are multiples
// of a's last place times 2^-24, that is of 2^-125 or more); a = 0 gives 0.  Five fused operations instead of a call of the general division
// with its reciprocal and its range test per element; the same bits (tests/test_division.py repeats the steps exactly).
constexpr float kDivMin = 3.30872245e-24f;
__device__ __forceinline__ float div_by(float a, float b, float y) {
    float q = a * y;
    q = fmaf(fmaf(-q, b, a), y, q);
    return fmaf(fmaf(-q, b, a), y, q);
}
// Four probabilities exp2f(x - mx) / denom of a group (y = the rounded 1 / denom).
__device__ __forceinline__ float4 prob4(float4 v, float mx, float denom, float y) {
    v.x = exp2f(v.x - mx); v.y = exp2f(v.y - mx); v.z = exp2f(v.z - mx); v.w = exp2f(v.w - mx);
    if (fminf(fminf(v.x, v.y), fminf(v.z, v.w)) >= kDivMin)
        return make_float4(div_by(v.x, denom, y), div_by(v.y, denom, y), div_by(v.z, denom, y), div_by(v.w, denom, y));
    return make_float4(v.x / denom, v.y / denom, v.z / denom, v.w / denom);
}

// Adds one group of a row of which nothing is cut off to a lane's ordered mass above the threshold (the smallest
// probability of the row) and counts its ties.
__device__ __forceinline__ void add_open(float4 v, float thr, float& gtp, uint32_t& eqk) {
    const float e[4] = {v.x, v.y, v.z, v.w};
    if (fminf(fminf(v.x, v.y), fminf(v.z, v.w)) > thr) {
#pragma unroll
        for (int i = 0; i < 4; i++) gtp += e[i];
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (e[i] > thr) gtp += e[i];
            else eqk++;
        }
    }
}
// Appends the candidates of one float4 group to the lane's list (rare; out of line).
__device__ __forceinline__ void append_candidates(float4 v, float beta_e, float* list, int stride4, int cap, int& nc, int& ns) {
    const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; j++) {
        if (e[j] >= beta_e) {
            if (nc < cap) list[(nc >> 2) * stride4 + (nc & 3)] = e[j];
            nc++;
            ns += (e[j] > beta_e) ? 1 : 0;
        }
    }
}


}  // namespace rs
