// Device functions shared by the router, grouping and glue kernels: the in-order sums of the
// reference (serial by definition) and the softmax top-k of one row.
#pragma once
#include "bitmath.cuh"
#include "internal.h"
#include "q4_core.cuh"

namespace sb {

static __device__ __forceinline__ void flag(int* status, int bit) {
    if (status) atomicOr(status, bit);
}

// Operations that stay where they are written: the compiler moved loads down to their uses and products to their adds,
// which a lone warp pays for with their whole latency.
static __device__ __forceinline__ float4 load_now(const float* p) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"((uint32_t)__cvta_generic_to_shared(p)));
    return v;
}
static __device__ __forceinline__ void add_now(float& a, float p) { asm volatile("add.rn.f32 %0, %0, %1;" : "+f"(a) : "f"(p)); }

// 0 + p[0] + p[1] + ... + p[n - 1], in order, by one warp on a scheduler of its own (all lanes alike).  p in shared memory,
// 16-byte aligned; n a positive multiple of 64.  32 terms are loaded between the adds of the 32 before them.
static __device__ __forceinline__ float chain_sum(const float* p, int n) {
    float4 a[8], b[8];
    float acc = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; i++) a[i] = load_now(p + 4 * i);
#pragma unroll 1
    for (int c = 0; c < n; c += 64) {
        const float* next = p + (c + 64 < n ? c + 64 : c);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            b[i] = load_now(p + c + 32 + 4 * i);
            add_now(acc, a[i].x); add_now(acc, a[i].y); add_now(acc, a[i].z); add_now(acc, a[i].w);
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
            a[i] = load_now(next + 4 * i);
            add_now(acc, b[i].x); add_now(acc, b[i].y); add_now(acc, b[i].z); add_now(acc, b[i].w);
        }
    }
    return acc;
}

// Serial sum of squares of one row, in element order, as the reference does
// (gemma4.c:46-62, src/text_verify_cpu.c:642-655).  The squares are formed in
// parallel beforehand; one thread then runs the add chain over them, reading
// shared memory 16 bytes at a time so the loads run ahead of the 4-cycle adds.
static __device__ __forceinline__ float serial_sum(const float* sq, int n) {
    float ss = 0.0f;
    int i = 0;
    if ((((uintptr_t)sq) & 15) == 0) {
#pragma unroll 4
        for (; i + 8 <= n; i += 8) {
            const float4 a = *(const float4*)(sq + i);
            const float4 b = *(const float4*)(sq + i + 4);
            ss = __fadd_rn(ss, a.x); ss = __fadd_rn(ss, a.y); ss = __fadd_rn(ss, a.z); ss = __fadd_rn(ss, a.w);
            ss = __fadd_rn(ss, b.x); ss = __fadd_rn(ss, b.y); ss = __fadd_rn(ss, b.z); ss = __fadd_rn(ss, b.w);
        }
    }
    for (; i < n; i++) ss = __fadd_rn(ss, sq[i]);
    return ss;
}

// The same sum - s = 0; s = fl(s + p[i]) for i = 0..n-1, bit for bit - by the whole block, for any terms.
//
// The terms are cut into 32 segments.  A chain of additions cannot be cut, but what a segment makes of its starting value can
// be tabulated: the segment's real additions are run from ORDERED_CANDS candidates, spaced by g around a predicted start,
// and the exact running sum then only has to pick its candidate, segment after segment.
//
//   1. sums in any order predict the running sum at every quarter of a segment.  In a second round the real additions of a
//      quarter from there add up to better predictions, as they leave out what the chain's roundings leave out: sums with
//      terms of both signs need them (half as many looks without an answer, below), squares do not;
//   2. lane t of three warps runs segment t from five or six candidates each, with g = the larger of ulp(start) and u / 8 (u: the unit
//      of the last place of the largest sum seen at the segment's quarters).  A fourth warp runs it from two sentinels well
//      outside the candidates and sees whether the two stay in the same binades, step by step, and in which at most.  As
//      additions are monotone, a path that starts between the sentinels then stays in those binades too;
//   3. the running sum s is start + q g.  Where q is one of -8 .. 7 the candidate IS s.  Otherwise the candidate 16 k g away
//      from s stands for it, if both lie between sentinels that stayed together and 16 g is an even number of units of the
//      last place everywhere in the segment: both paths then round alike, half-way cases too, and stay 16 k g apart;
//   4. one warp per four segments makes a table of them together (its candidates are the first one's, and so are its
//      sentinels, which must pass between the sentinels of the others); one warp walks the eight tables from s = 0.  Where a
//      table has no answer it takes the four segments one by one, and where a segment has none, term by term.
// So the predictions decide only how much runs side by side: every result is a real addition of the chain, or one shifted
// by an amount that is proven to pass through it.  Just under 1 % of the segments of a router row have no answer (mostly
// where the sum passes zero and its binade changes with every step), hardly any of squares.  The sixth such segment takes the
// rest of the chain with it, so that terms of which nothing can be tabulated (pairs that cancel) take at most half as long again
// as a chain: 2816 of them 17 400 cycles, 26 500 without that limit, 12 100 as a chain by one warp.
// What bounds it: the additions of 2 (n / 32 dependent ones, six side by side, about 10 cycles each), those of segments
// without an answer (600 cycles each with what it takes to get there), 60 to 130 cycles per look into a table, five or six barriers
// with a scan or two between them.  Measured in a block of 640 threads (B200): 2816 squares 4000 cycles, where integer increments
// between the points at which the sum changes its binade took 7500; 2816 products 5200 on average, where one warp's chain took
// 13 700; 5120 of them 5800 (25 000).  32 candidates with more warps, or one segment per warp with a candidate per lane, were
// slower: loads of the terms took the time.
//
// p and scratch (ORDERED_SCRATCH words): shared memory, 16-byte aligned; p written by the block, no barrier needed before the
// call.  At least 256 threads, whole warps; every thread of the block must call; all return the sum.
constexpr int ORDERED_CANDS = 16;
constexpr int ORDERED_MISSES = 6;                         // segments without an answer, the last of them with all that follow
constexpr int ORDERED_PITCH = 20;                         // floats per table: candidates' ends, the sentinels', bank offset
constexpr int ORDERED_GROUP = 4, ORDERED_GROUPS = 32 / ORDERED_GROUP;
constexpr int ORDERED_SCRATCH = 8 + 2 * 4 * 32 + 4 * 32 + 2 * 32 + 32 + 2 * ORDERED_GROUPS + (32 + ORDERED_GROUPS) * ORDERED_PITCH;

static __device__ __forceinline__ uint32_t shared_at(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
static __device__ __forceinline__ float4 shared_f4(uint32_t at) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at));
    return v;
}
static __device__ __forceinline__ float2 shared_f2(uint32_t at) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(at));
    return v;
}
static __device__ __forceinline__ float shared_f(uint32_t at) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at));
    return v;
}

// term(v.x), term(v.y), ... for the `mine` pieces of four floats at `at` and zeros up to a multiple of four of `pieces` or
// more: four pieces are loaded while the four before them are used.  The same trips for all lanes and no branch inside: lanes
// that part company in a loop are slow to meet again, and one by one they take 32 times as long.
template <class Term>
static __device__ __forceinline__ void for_terms(uint32_t at, uint32_t zeros, int mine, int pieces, Term term) {
    float4 a[4];
#pragma unroll
    for (int j = 0; j < 4; j++) a[j] = shared_f4(j < mine ? at + 16 * j : zeros);
#pragma unroll 2
    for (int i = 0; i < pieces; i += 4) {
        float4 b[4];
#pragma unroll
        for (int j = 0; j < 4; j++) b[j] = shared_f4(i + 4 + j < mine ? at + 16 * (i + 4 + j) : zeros);
#pragma unroll
        for (int j = 0; j < 4; j++) { term(a[j].x); term(a[j].y); term(a[j].z); term(a[j].w); }
#pragma unroll
        for (int j = 0; j < 4; j++) a[j] = b[j];
    }
}

// ulp of a float with these exponent bits (0x7f800000 & bits); 0 where that is no normal number
static __device__ __forceinline__ float ulp_of(uint32_t exponent) {
    return exponent > (23u << 23) ? __uint_as_float(exponent - (23u << 23)) : 0.0f;
}
static __device__ __forceinline__ uint32_t exponent_of(float v) { return __float_as_uint(v) & 0x7f800000u; }

// A look into one table: seg = start, g, 1 / g; between = sentinels (none: empty).  s becomes the sum behind the segment.
// inside: s has to lie between the sentinels even where it is a candidate.  No branches.
static __device__ __forceinline__ bool ordered_step(float& s, const float4& seg, const float2& between, uint32_t ends, bool inside) {
    constexpr float MAGIC = 12582912.0f + ORDERED_CANDS / 2;          // q + MAGIC has q + CANDS / 2 in its low bits
    const float d = __fsub_rn(s, seg.x), m = __fmaf_rn(d, seg.z, MAGIC);
    const uint32_t k = __float_as_uint(m) & (ORDERED_CANDS - 1);
    const float end = shared_f(ends + 4 * k);
    const float from = __fmaf_rn(__fsub_rn(__uint_as_float(0x4b000000u | k), 8388608.0f + ORDERED_CANDS / 2), seg.y, seg.x);
    const float shift = __fsub_rn(s, from);
    const int in = (int)(between.x <= s) & (int)(s <= between.y);
    const int whole = (int)(__fsub_rn(m, MAGIC) == __fmul_rn(d, seg.z));
    s = __fadd_rn(end, shift);
    return ((int)(shift == 0.0f) | (in & whole)) & (in | (int)!inside) & (int)(s == s);
}

// The same sum, in one chain, by warp `who` (blocks of an SM that take different warps add on different schedulers).  scratch:
// CHAIN_SCRATCH words are enough.
constexpr int CHAIN_SCRATCH = 8;
static __device__ __forceinline__ float block_sum_chain(const float* p, int n, uint32_t* scratch, int who) {
    float* const result = (float*)scratch + 4;              // where the pieces leave theirs, too
    __syncthreads();
    if ((int)(threadIdx.x >> 5) == who) {
        float s = n >= 64 ? chain_sum(p, n & ~63) : 0.0f;
        for (int i = n & ~63; i < n; i++) s = __fadd_rn(s, p[i]);
        if ((threadIdx.x & 31) == 0) *result = s;
    }
    __syncthreads();
    return *result;
}

// Terms up to which that is the shorter way for a block by itself: the pieces cost 2800 (squares) or 3700 cycles (products)
// whatever their length, a chain 460 and 4.15 a term.  Block of 640 threads, chain / pieces: 576 squares 2860 / 2990, 640 3120 /
// 2990; 768 products 3650 / 4370, 832 3910 / 4010, 896 4180 / 4140.
static __host__ __device__ __forceinline__ bool sum_in_chain(int n, int rounds) { return n <= (rounds == 1 ? 576 : 832); }

static __device__ __forceinline__ float block_sum_ordered(float* p, int n, int rounds, uint32_t* scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // words of scratch: zeros [4], result [4], sums of the segments' quarters [2][4][32], seg [32] (start, g, 1 / g, first piece << 16 | pieces), sentinels
    // [32][2], largest unit of the last place [32], sentinels of the groups [GROUPS][2], ends [32][PITCH], of groups [GROUPS][PITCH]
    constexpr int RESULT = 4, QUARTER = 8, SEG = QUARTER + 2 * 4 * 32, BETWEEN = SEG + 4 * 32, UNIT = BETWEEN + 2 * 32, GBETWEEN = UNIT + 32,
                  ENDS = GBETWEEN + 2 * ORDERED_GROUPS, GENDS = ENDS + 32 * ORDERED_PITCH;
    static_assert(GENDS + ORDERED_GROUPS * ORDERED_PITCH == ORDERED_SCRATCH && ENDS % 4 == 0 && SEG % 4 == 0, "scratch");
    float* const sf = (float*)scratch;
    const uint32_t base = shared_at(scratch), zeros = base, terms = shared_at(p);
    // segments of an odd number of 16-byte pieces: the lanes read other banks
    const int pieces = ((n + 127) >> 7) | 1, all = (n + 3) >> 2;
    if (threadIdx.x < 4) {
        sf[threadIdx.x] = 0.0f;
        if (n + (int)threadIdx.x < 4 * all) p[n + threadIdx.x] = 0.0f;
    }
    __syncthreads();
    // ---- 1. predictions: sums of the segments' quarters, from zero and then from where those predict them to start
    float q0, q1, q2, q3, start;                          // the segment's quarters, summed up; its start
    auto predict = [&](int table) {
        const float* q = sf + QUARTER + 128 * table + lane;
        q0 = q[0]; q1 = q0 + q[32]; q2 = q1 + q[64]; q3 = q2 + q[96];
        start = q3;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float t = __shfl_up_sync(0xffffffffu, start, o);
            start += lane >= o ? t : 0.0f;
        }
        start = __shfl_up_sync(0xffffffffu, start, 1);
        start = lane == 0 ? 0.0f : start;
    };
    const int quarter = (pieces + 3) >> 2;
#pragma unroll 1
    for (int table = 0; table < rounds; table++) {
        if (warp < 4) {
            float r0 = 0.0f;
            if (table != 0) {
                predict(0);
                r0 = start + (warp < 2 ? (warp == 0 ? 0.0f : q0) : (warp == 2 ? q1 : q2));
            }
            const int first = lane * pieces + warp * quarter;
            float r = r0;
            for_terms(terms + 16 * first, zeros, min(all - first, min(quarter, pieces - warp * quarter)), quarter, [&](float t) { r = __fadd_rn(r, t); });
            sf[QUARTER + 128 * table + 32 * warp + lane] = r - r0;
        }
        __syncthreads();
    }
    // ---- 2. candidates and sentinels
    if (warp < 4) {
        predict(rounds - 1);
        // a segment that would start far below the values it reaches has no good candidates: it starts a quarter later
        const float inner = fmaxf(fmaxf(fabsf(start + q0), fabsf(start + q1)), fmaxf(fabsf(start + q2), fabsf(start + q3)));
        const bool late = lane > 0 && fabsf(start) < 0.125f * inner && fabsf(start) < fabsf(start + q0);
        const uint32_t lates = __ballot_sync(0xffffffffu, late) >> lane;
        const int begin = lane * pieces + (lates & 1u ? quarter : 0);
        const int count = min(lane * pieces + pieces + (lates & 2u ? quarter : 0), all) - begin, trips = (int)__reduce_max_sync(0xffffffffu, (unsigned)max(count, 0));
        start = late ? start + q0 : start;
        const float next = __shfl_down_sync(0xffffffffu, start, 1);
        const float u = ulp_of(exponent_of(fmaxf(inner, fmaxf(fabsf(start), lane < 31 ? fabsf(next) : 0.0f))));
        const uint32_t from = terms + 16 * begin;
        float g = fmaxf(ulp_of(exponent_of(start)), u * (2.0f / ORDERED_CANDS));
        g = g >= 1.0e-36f && g <= 1.0e36f ? g : 0.0f;     // 1 / g is exact: g is a power of two
        if (warp < 3) {
            static_assert(ORDERED_CANDS == 16, "candidates 0..5, 5..10, 10..15: a scheduler each, the sentinels on the fourth");
            float s[6];
#pragma unroll
            for (int i = 0; i < 6; i++) s[i] = __fmaf_rn((float)(5 * warp + i - ORDERED_CANDS / 2), g, start);
            for_terms(from, zeros, count, trips, [&](float t) {
#pragma unroll
                for (int i = 0; i < 6; i++) s[i] = __fadd_rn(s[i], t);
            });
#pragma unroll
            for (int i = 0; i < 6; i++) sf[ENDS + lane * ORDERED_PITCH + 5 * warp + i] = s[i];
        } else {
            // 128 u: several times what the roundings of a few thousand terms add up to, a small part of a binade.  Those that
            // have to pass between the sentinels of the segments behind start closer.
            const float w = lane % ORDERED_GROUP == 0 ? (rounds == 1 ? 64.0f : 32.0f) : 128.0f, lo0 = start - w * u, hi0 = start + w * u;
            float lo = lo0, hi = hi0, top = fabsf(hi0);
            uint32_t differ = __float_as_uint(lo) ^ __float_as_uint(hi);
            for_terms(from, zeros, count, trips, [&](float t) {
                lo = __fadd_rn(lo, t);
                hi = __fadd_rn(hi, t);
                differ |= __float_as_uint(lo) ^ __float_as_uint(hi);
                top = fmaxf(top, fabsf(hi));
            });
            const float most = ulp_of(exponent_of(top));
            const bool together = (differ & 0xff800000u) == 0u && exponent_of(top) != 0x7f800000u && most > 0.0f && g * ORDERED_CANDS >= 2.0f * most;
            *(float4*)(sf + SEG + 4 * lane) = make_float4(start, g, g > 0.0f ? __uint_as_float(0x7f000000u - __float_as_uint(g)) : 0.0f, __int_as_float(begin << 16 | max(count, 0)));
            *(float2*)(sf + BETWEEN + 2 * lane) = together ? make_float2(lo0, hi0) : make_float2(1.0f, -1.0f);
            sf[UNIT + lane] = together ? most : __uint_as_float(0x7f800000u);
            *(float2*)(sf + ENDS + lane * ORDERED_PITCH + ORDERED_CANDS) = make_float2(lo, hi);
        }
    }
    __syncthreads();
    // ---- 3. tables of four segments
    if (warp < ORDERED_GROUPS) {
        const int t0 = warp * ORDERED_GROUP, k = min(lane, ORDERED_CANDS + 1);
        const bool sentinel = lane >= ORDERED_CANDS;
        const uint32_t at = base + 4 * (SEG + 4 * t0), bt = base + 4 * (BETWEEN + 2 * t0), et = base + 4 * (ENDS + t0 * ORDERED_PITCH);
        float s = shared_f(et + 4 * k);
        float4 seg[ORDERED_GROUP];
        float2 between[ORDERED_GROUP];
#pragma unroll
        for (int i = 0; i < ORDERED_GROUP; i++) {
            seg[i] = shared_f4(at + 16 * i);
            between[i] = shared_f2(bt + 8 * i);
        }
        const float4 unit = shared_f4(base + 4 * (UNIT + t0));
        int ok = (int)!sentinel | (int)(between[0].x <= between[0].y);
#pragma unroll
        for (int i = 1; i < ORDERED_GROUP; i++) ok &= (int)ordered_step(s, seg[i], between[i], et + 4 * ORDERED_PITCH * i, sentinel);
        const float most = fmaxf(fmaxf(unit.x, unit.y), fmaxf(unit.z, unit.w));
        const bool together = __all_sync(0xffffffffu, ok | (int)!sentinel) && seg[0].y * ORDERED_CANDS >= 2.0f * most;
        if (lane < ORDERED_CANDS) sf[GENDS + warp * ORDERED_PITCH + lane] = ok ? s : __uint_as_float(0x7fffffffu);
        if (lane == 0) *(float2*)(sf + GBETWEEN + 2 * warp) = together ? between[0] : make_float2(1.0f, -1.0f);
    }
    __syncthreads();
    // ---- 4. the walk.  Squares: as if every look had its answer.  Else, and if one has not: what the next look needs is loaded
    // while this one waits for its table
    if (threadIdx.x == 0) {
        float s = 0.0f;
        bool all_known = rounds == 1;
        if (rounds == 1) {
#pragma unroll
            for (int i = 0; i < ORDERED_GROUPS; i++)
                all_known &= ordered_step(s, shared_f4(base + 4 * (SEG + 4 * ORDERED_GROUP * i)), shared_f2(base + 4 * (GBETWEEN + 2 * i)),
                                          base + 4 * (GENDS + i * ORDERED_PITCH), false);
            if (!all_known) s = 0.0f;
        }
        float4 seg = shared_f4(base + 4 * SEG);
        float2 lohi = shared_f2(base + 4 * GBETWEEN);
        int missed = 0;
#pragma unroll 1
        for (int i = all_known ? ORDERED_GROUPS : 0; i < ORDERED_GROUPS; i++) {
            const int t0 = ORDERED_GROUP * i, n0 = min(t0 + ORDERED_GROUP, 31), ni = min(i + 1, ORDERED_GROUPS - 1);
            const float4 next_seg = shared_f4(base + 4 * (SEG + 4 * n0));
            const float2 next_lohi = shared_f2(base + 4 * (GBETWEEN + 2 * ni));
            float after = s;
            if (!ordered_step(after, seg, lohi, base + 4 * (GENDS + i * ORDERED_PITCH), false)) {
                float2 own = shared_f2(base + 4 * (BETWEEN + 2 * t0));
#pragma unroll 1
                for (int t = t0; t < t0 + ORDERED_GROUP; t++) {
                    const float4 one_seg = shared_f4(base + 4 * (SEG + 4 * min(t + 1, 31)));
                    const float2 one_own = shared_f2(base + 4 * (BETWEEN + 2 * min(t + 1, 31)));
                    after = s;
                    if (!ordered_step(after, seg, own, base + 4 * (ENDS + t * ORDERED_PITCH), false)) {
                        after = s;
                        missed++;
                        const int at = __float_as_int(seg.w), first = at >> 16;
                        int count = at & 0xffff;
                        if (missed >= ORDERED_MISSES) {              // the rest of the chain
                            count = all - first;
                            t = 31;
                            i = ORDERED_GROUPS;
                        }
                        for_terms(terms + 16 * first, zeros, count, count, [&](float v) { after = __fadd_rn(after, v); });
                    }
                    s = after;
                    seg = one_seg;
                    own = one_own;
                }
            }
            s = after;
            seg = next_seg;
            lohi = next_lohi;
        }
        sf[RESULT] = s;
    }
    __syncthreads();
    return sf[RESULT];
}

// Softmax top-k (gemma4.c:132-186) + ascending-expert ordering of the selected
// pairs (gemma4_text.c:8541-8550).  The insertion top-k with strict '>' equals
// ranking by (logit descending, expert ascending); the softmax denominator and
// the renormalisation sum are serial chains in expert / rank order.
//
// Executed by a group of `gsize` >= 64 consecutive threads (ltid = index in group, whole warps) on one row; every thread of
// the block must call it (block-wide barriers inside), groups without a row pass active = false.  logit(e): the row's logit of
// expert e, the same at every call.  sm = this group's scratch of 2E + 2*topk floats (16-byte aligned), sc = 4 floats of
// per-group scalars, bar: number of a barrier of the group's own (1 and up).
//
// Nothing but latencies: up to 128 experts the group's first warp picks the selections, the largest of four keys per lane
// at a time, while the other warps evaluate the exponentials and the second one adds them in order; then the first warp does
// the rest, a selection per lane (the divisions side by side, the sum of the selected ones by all lanes alike).
// Measured in a decode layer (128 experts, top-8): from the logits in the block to the weights 3500 cycles, 5000 with the sum after
// the selections and one thread reading each selection back; the exponentials and their 128 ordered additions take 1600 of them.
static __device__ __forceinline__ void group_barrier(int bar, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(threads) : "memory"); }

template <class Logit>
static __device__ __forceinline__ void topk_group(bool active, Logit logit, const float* per_expert_scale, int32_t* sel_out, float* w_out,
                                                  int E, int topk, int sort_by_expert, int* status, float* sm, float* sc,
                                                  int ltid, int gsize, int bar) {
    constexpr int KEYS = 4;          // experts per lane of the first warp
    float* sl = sm;                  // [E] logits (more than 32 * KEYS experts)
    float* se = sm + E;              // [E] exp(l - max)
    int* ssel = (int*)(sm + 2 * E);  // [topk]
    float* sw = sm + 2 * E + topk;   // [topk]
    int* s_bad = (int*)(sc + 3);
    const bool few = E <= 32 * KEYS;
    float own = 0.0f;                // the first expert whose exponential this thread evaluates
    if (active && few && ltid >= 32 && ltid - 32 < E) own = logit(ltid - 32);
    uint32_t key[KEYS];
    int mine = 0;                    // first warp: selection number ltid
    if (active && ltid < 32) {
        float m = __int_as_float(0xff800000);
        bool bad = false;
        if (few) {
#pragma unroll
            for (int i = 0; i < KEYS; i++) {
                const int e = ltid + 32 * i;
                key[i] = 0u;                                     // below every finite logit's key
                if (e < E) {
                    const float v = logit(e);
                    bad |= !finite_f(v) || (per_expert_scale && !finite_f(per_expert_scale[e]));
                    m = fmaxf(m, v);
                    const uint32_t b = __float_as_uint(__fadd_rn(v, 0.0f));      // -0 ranks like +0
                    key[i] = (b & 0x80000000u) ? ~b : b | 0x80000000u;
                }
            }
        } else {
            for (int e = ltid; e < E; e += 32) {
                const float v = logit(e);
                bad |= !finite_f(v) || (per_expert_scale && !finite_f(per_expert_scale[e]));
                m = fmaxf(m, v);
                sl[e] = v;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        bad = __any_sync(0xffffffffu, bad);
        if (ltid == 0) {
            sc[0] = m;
            *s_bad = bad ? 1 : 0;
        }
        __syncwarp();
    }
    __syncthreads();
    // the reference rejects non-finite logits before ranking (gemma4.c:149-152)
    const bool go = active && !*s_bad;
    if (go && !few) {
        const float mx = sc[0];
        for (int e = ltid; e < E; e += gsize) {
            const float v = sl[e];
            se[e] = expf_exact(__fsub_rn(v, mx));
            int rank = 0;
            for (int o = 0; o < E; o++) {
                const float u = sl[o];
                rank += (u > v || (u == v && o < e)) ? 1 : 0;
            }
            if (rank < topk) ssel[rank] = e;
        }
    } else if (go && ltid >= 32) {
        const float mx = sc[0];
        for (int e = ltid - 32; e < E; e += gsize - 32)
            se[e] = expf_exact(__fsub_rn(e == ltid - 32 ? own : logit(e), mx));
        group_barrier(bar, gsize - 32);
        if (ltid < 64) {
            const float all = (E & 63) == 0 && (((uintptr_t)se) & 15) == 0 ? chain_sum(se, E) : serial_sum(se, E);
            if (ltid == 32) sc[1] = all;
        }
    } else if (go) {
#pragma unroll 1
        for (int j = 0; j < topk; j++) {
            uint32_t best = key[0];
#pragma unroll
            for (int i = 1; i < KEYS; i++) best = max(best, key[i]);
            best = __reduce_max_sync(0xffffffffu, best);
            int e = 0;                                           // the lowest expert of those that tie
#pragma unroll
            for (int i = KEYS - 1; i >= 0; i--) {
                const uint32_t tied = __ballot_sync(0xffffffffu, key[i] == best);
                e = tied ? 32 * i + __ffs(tied) - 1 : e;
            }
#pragma unroll
            for (int i = 0; i < KEYS; i++) key[i] = e == ltid + 32 * i ? 0u : key[i];
            mine = j == ltid ? e : mine;
            if (topk > 32 && ltid == 0) ssel[j] = e;
        }
    }
    __syncthreads();
    if (go && ltid < 32) {
        float all;
        if (few) all = sc[1];
        else all = (E & 63) == 0 && (((uintptr_t)se) & 15) == 0 ? chain_sum(se, E) : serial_sum(se, E);
        bool bad = !(all > 0.0f) || !finite_f(all);
        if (few && topk <= 32) {
            const float w = __fdiv_rn(se[mine], all);
            float selsum = 0.0f;
            int before = 0;
#pragma unroll 4
            for (int j = 0; j < topk; j++) {
                selsum = __fadd_rn(selsum, __shfl_sync(0xffffffffu, w, j));
                before += __shfl_sync(0xffffffffu, mine, j) < mine ? 1 : 0;
            }
            if (!(selsum > 0.0f) || !finite_f(selsum)) bad = true;
            if (ltid < topk) {
                const int pos = sort_by_expert ? before : ltid;
                sel_out[pos] = mine;
                w_out[pos] = __fmul_rn(__fdiv_rn(w, selsum), per_expert_scale ? per_expert_scale[mine] : 1.0f);
            }
        } else {
            for (int j = ltid; j < topk; j += 32) sw[j] = __fdiv_rn(se[ssel[j]], all);
            __syncwarp();
            float selsum = 0.0f;
#pragma unroll 8
            for (int j = 0; j < topk; j++) selsum = __fadd_rn(selsum, sw[j]);
            if (!(selsum > 0.0f) || !finite_f(selsum)) bad = true;
            for (int j = ltid; j < topk; j += 32) {
                const int e = ssel[j];
                const float nrm = __fdiv_rn(sw[j], selsum);
                const float w = __fmul_rn(nrm, per_expert_scale ? per_expert_scale[e] : 1.0f);
                int pos = j;
                if (sort_by_expert) {
                    pos = 0;
#pragma unroll 8
                    for (int i = 0; i < topk; i++) pos += (ssel[i] < e) ? 1 : 0;
                }
                sel_out[pos] = e;
                w_out[pos] = w;
            }
        }
        if (ltid == 0 && bad) *s_bad = 1;
    }
    if (active && ltid == 0 && *s_bad) flag(status, SB_ERR_NONFINITE);
}

static __host__ __device__ __forceinline__ int topk_scratch_floats(int E, int topk) {
    return ((2 * E + 2 * topk + 3) & ~3) + 4;
}

}  // namespace sb
