// Grouped affine-Q4 expert GEMMs on the 5th-generation tensor cores (tcgen05 + TMEM) for prefill-sized token groups.
// TOLERANCE path: fp16 operands, fp32 accumulation in TMEM.  The bit-exact kernels in batch_kernels.cu and q4_kernels.cu
// remain the reference-conformant path.
//
// Two precisions (template SPLIT):
//   single  weights dequantised as q*s+b and rounded to fp16, activations rounded to fp16: max |err| about 5e-4 to
//           7e-4 of the row maximum
//   split   x * (q s + b) = x * (q - 8) s + x * (b + 8 s).  (q - 8) s has at most 4 + 8 significant bits, so it is EXACT
//           in fp16 once the row is scaled by a power of two (q4_tc_tables_kernel) that keeps it in range; b + 8 s is
//           constant over a quantisation group, so its part of the sum is a second, 64 times shorter contraction of the
//           groups' means of x with c = b + 8 s (hi + lo halves): one or a few "correction" chunks after the ordinary
//           ones.  Activations are hi + lo halves (lo = fp16(x - hi)).  So a K step takes two products, Xh W and Xl W,
//           instead of three with split weights, and a stage holds one weight tile, not two: max |err| 1.6e-5 of the row
//           maximum, from the halves of x.  Passes of up to 64 tokens put the hi and the lo rows into ONE 128-row tile
//           (sixteen hi rows, then their lo rows, in every quarter) and take a single MMA; the epilogue adds the two.
//
// A unit of work = one 128-token pass of one tile of weight rows of one expert group.  A small kernel writes the layer's
// units into a work list from the grouped jobs (pass and tile counts are only known on the device); one resident block per
// SM draws units from it with an atomic counter until it is empty, its pipeline running on from one unit into the next.
// Grids of one block per tile paid for every block's launch with 225 KB of shared memory, for the empty blocks of experts
// with fewer passes than the grid allowed, and for experts with several hundred tokens finishing last.
// The tokens of a pass (stale rows above them) are the MMA's M side, read from shared memory as they arrive by TMA; 256
// weight rows are the N side, dequantised into a K-major 128-byte-swizzled stage.  The 256 rows are one tile of the down
// matrix, or - fused - 128 rows of gate followed by the same 128 rows of up: one instruction is M128 x N256 x K16, and the
// GeGLU pairs accumulator column c with 128 + c.  Accumulators: lane = token, column = weight row, double-buffered by unit.
// K advances in 64-column chunks = one quantisation group per row.
//   weight thread     draws the unit and passes it to the other roles through a shared-memory ring; loads packed nibbles
//                     (tiled TMA over the expert pool: bytes x rows x experts) into a ring of four 8 KB slots
//   token thread      loads the tokens' fp16 rows (128-byte swizzle) into a ring of three or four tiles.  A ring of its
//                     own: a packed slot is free as soon as its bytes are in registers, a token tile only after its MMAs
//   converter warps   two groups of eight warps on alternate chunks (thread = stage row): packed bytes -> registers ->
//                     fp16 -> the stage; the row's (scale << 16) | bias word comes straight from global memory a chunk
//                     pair ahead; one mbarrier arrival per warp
//   issuer thread     tcgen05.mma.kind::f16 of every converted chunk, tcgen05.commit on the chunk's "done" barrier; polls
//                     the next chunk's barriers before issuing, so the answer arrives behind the MMAs
//   epilogue          all converter warps tcgen05.ld the accumulators of a unit (warp w: lane quarter w % 4, a quarter of
//                     the columns), sixteen columns at a time to stay inside 96 registers: GeGLU (fused gate/up) or plain
//                     store (down).  It runs after the group's second chunk of the NEXT unit, so that the tensor core
//                     does not drain at a unit's end
// Measured (B200, 1965 MHz, a whole layer with its router: hidden 2816, inter 704, 128 experts, top-8): 512 tokens in split
// precision 800 us with three MMAs per K step on split weights -> 515 with exact weights and separate rings -> 473 with the
// delayed epilogue, four stages and the correction chunk's table words loaded at once (they came in four serial batches, 9000
// cycles a chunk) -> 430 with cheaper kernels around the GEMMs and tables by group -> 420 with whole sectors per store and
// half a stage for a last tile of 64 rows (gate/up 201, down 107).  1999 tokens in single precision 780 -> 707 -> 694 -> 607
// -> 585 (gate/up 222, down 142).  The tensor pipe is busy 36 to 49 % of the time, the schedulers issue in 47 to 62 % of the
// cycles: converters and tensor core still wait for one another.
// What was measured on the way here: a register ring of global loads for the packed bytes does not prefetch - waiting for
// the oldest load also waits for the younger ones that share its scoreboard (hence TMA); one mbarrier wait costs 150 to 250
// cycles even when its phase is complete, so the phases needed next are tested ahead; a tcgen05.mma costs the issuing
// thread about 100 cycles for any N <= 128 (weights on M, from shared memory or from tensor memory: both forms ran 8 such
// instructions per fused chunk), so the weights sit on N, 256 rows per instruction.
// Column order inside every group of 8 K columns is permuted to [0,4,1,5,2,6,3,7] in BOTH operands (a contraction does not
// care): it is the order in which two masks and one shift peel half2 pairs out of a packed 32-bit word.
// Every mbarrier wait is bounded: on expiry the block raises a shared flag, records an error in the status word, every role
// leaves its loop, outstanding copies and MMAs are waited for (bounded), TMEM is freed and the block returns.
#include <cuda_fp16.h>

#include <stdlib.h>
#include <algorithm>
#include "internal.h"
#include "mbar.cuh"
#include "umma.cuh"
#include "q4_core.cuh"

namespace sb {

constexpr int TC_GROUP = 256;                // converter threads of one chunk (two groups take alternate chunks)
constexpr int TC_CONVERTERS = 2 * TC_GROUP;
constexpr int TC_THREADS = TC_CONVERTERS + 96;   // + issuer, weight and token warps
constexpr int TC_ISSUER_WARP = TC_CONVERTERS / 32, TC_WEIGHT_WARP = TC_ISSUER_WARP + 1, TC_TOKEN_WARP = TC_ISSUER_WARP + 2;
constexpr int TC_KC = 64;                    // K columns per chunk
constexpr uint32_t TC_TMEM_COLS = 512;
constexpr int TC_PK_BYTES = 128 * TC_KC / 2; // packed chunk of 128 rows (one matrix' share of a fused stage)
constexpr int TC_MAX_NT = 128;
constexpr int TC_MAX_SLOTS = 4;              // packed chunks in flight
// Entries of the ring through which the thread that draws the units passes them to the other roles.  It is at most
// TC_MAX_SLOTS chunks, i.e. units, ahead of the converters, and no role is more than three chunks and a unit behind
// those, so 16 entries are never overrun and need no "free" barrier.
constexpr int TC_ITEM_RING = 16;
constexpr int TC_SMEM_BYTES = 225 * 1024;    // dynamic shared memory of every launch (one block per SM)

// kind::f16 instruction descriptor: D = F32, A = B = F16, both K-major.
__device__ __forceinline__ uint32_t umma_idesc_f16(int M, int N) {
    return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// half2 {lo, hi} from two floats (round to nearest even)
__device__ __forceinline__ uint32_t f16x2_from(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ float f16_lo_to_f32(uint32_t h2) {
    float f;
    asm("{\n\t.reg .f16 l, h;\n\tmov.b32 {l, h}, %1;\n\tcvt.f32.f16 %0, l;\n\t}\n" : "=f"(f) : "r"(h2));
    return f;
}
__device__ __forceinline__ float f16_hi_to_f32(uint32_t h2) {
    float f;
    asm("{\n\t.reg .f16 l, h;\n\tmov.b32 {l, h}, %1;\n\tcvt.f32.f16 %0, h;\n\t}\n" : "=f"(f) : "r"(h2));
    return f;
}
__device__ __forceinline__ uint32_t hsub2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t hfma2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}

// Position of original column o (0..7) inside its group of 8 in the operands' K order
// [0,4,1,5,2,6,3,7].
__host__ __device__ __forceinline__ int tc_kpos(int o) { return ((o & 3) << 1) | (o >> 2); }

// Can q*s+b of this group be formed in fp16 arithmetic without loss?  s/16 and b must be
// exact fp16 values (bf16 has 8 significant bits) and 15*s+b must stay finite.
// bf16 exponent fields: s in [2^-13, 2^10), b zero or in [2^-17, 2^14).
__device__ __forceinline__ bool fp16_path_ok(uint32_t s_bits, uint32_t b_bits) {
    const uint32_t es = (s_bits >> 7) & 0xffu, eb = (b_bits >> 7) & 0xffu;
    const bool s_ok = es >= 114u && es <= 136u;
    const bool b_ok = (b_bits & 0x7fffu) == 0u || (eb >= 110u && eb <= 140u);
    return s_ok && b_ok;
}

// 32 consecutive Q4 elements of one row (16 packed bytes) -> 16 half2 words in the operands' K order
// (word 4 i + k holds columns (k, k + 4) of the i-th group of 8), fp16 arithmetic: a nibble masked in place
// under the exponent of 2^10 reads as 1024 + q (low nibble of a byte) or 1024 + 16 q (high nibble);
// subtracting 1024 is exact and one half2 fma with s (or s/16) forms q*s + b with a single rounding.
__device__ __forceinline__ void dequant_half_chunk_f16(const uint4& p, uint32_t s_bits, uint32_t b_bits,
                                                       uint32_t (&o)[16]) {
    const float s = bf16_bits_to_f32(s_bits), b = bf16_bits_to_f32(b_bits);
    const uint32_t s2 = f16x2_from(s, s), s2_16 = f16x2_from(s * 0.0625f, s * 0.0625f), b2 = f16x2_from(b, b);
    const uint32_t w[4] = {p.x, p.y, p.z, p.w};
    const uint32_t k1024 = 0x64006400u;
#pragma unroll
    for (int i = 0; i < 4; i++) {  // word i = 8 columns
        const uint32_t w0 = w[i], w1 = w[i] >> 8;
        uint32_t a0, a1, a2, a3;
        asm("lop3.b32 %0, %1, 0x000f000f, %2, 0xEA;" : "=r"(a0) : "r"(w0), "r"(k1024));   // cols (0,4)
        asm("lop3.b32 %0, %1, 0x00f000f0, %2, 0xEA;" : "=r"(a1) : "r"(w0), "r"(k1024));   // cols (1,5) * 16
        asm("lop3.b32 %0, %1, 0x000f000f, %2, 0xEA;" : "=r"(a2) : "r"(w1), "r"(k1024));   // cols (2,6)
        asm("lop3.b32 %0, %1, 0x00f000f0, %2, 0xEA;" : "=r"(a3) : "r"(w1), "r"(k1024));   // cols (3,7) * 16
        o[4 * i + 0] = hfma2(hsub2(a0, k1024), s2, b2);
        o[4 * i + 1] = hfma2(hsub2(a1, k1024), s2_16, b2);
        o[4 * i + 2] = hfma2(hsub2(a2, k1024), s2, b2);
        o[4 * i + 3] = hfma2(hsub2(a3, k1024), s2_16, b2);
    }
}

// The same 32 elements through fp32 (any scale).
__device__ __forceinline__ void dequant_half_chunk_f32(const NibbleMagic& mg, const uint4& p, uint32_t s_bits,
                                                       uint32_t b_bits, uint32_t (&o)[16]) {
    const float s = bf16_bits_to_f32(s_bits), b = bf16_bits_to_f32(b_bits);
    const uint32_t w[4] = {p.x, p.y, p.z, p.w};
    const f32x2 ss = pack2(s, s), bb = pack2(b, b);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        f32x2 q[4];
        nibbles4(w[i] & 0xffffu, mg, q[0], q[1]);
        nibbles4(w[i] >> 16, mg, q[2], q[3]);
        float v[8];
#pragma unroll
        for (int k = 0; k < 4; k++) unpack2(fma2(q[k], ss, bb), v[2 * k], v[2 * k + 1]);
#pragma unroll
        for (int k = 0; k < 4; k++) o[4 * i + k] = f16x2_from(v[k], v[k + 4]);   // half2 k holds columns (k, k + 4)
    }
}

__device__ __forceinline__ uint32_t hmul2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

// Hi + lo precision: (q - 8) * s of 32 elements.  q - 8 has three bits and s eight, so the fp16 product is exact: no lo
// half of the weights is needed; what is left of w = (q - 8) s + c, c = b + 8 s, is constant in a group and goes through
// the correction chunks.
__device__ __forceinline__ void dequant_exact(const uint4& p, uint32_t s2, uint32_t s2_16, uint32_t (&o)[16]) {
    const uint32_t w[4] = {p.x, p.y, p.z, p.w};
    const uint32_t k1024 = 0x64006400u, k1032 = 0x64086408u, k1152 = 0x64806480u;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t w0 = w[i], w1 = w[i] >> 8;
        uint32_t a0, a1, a2, a3;
        asm("lop3.b32 %0, %1, 0x000f000f, %2, 0xEA;" : "=r"(a0) : "r"(w0), "r"(k1024));   // cols (0,4)
        asm("lop3.b32 %0, %1, 0x00f000f0, %2, 0xEA;" : "=r"(a1) : "r"(w0), "r"(k1024));   // cols (1,5) * 16
        asm("lop3.b32 %0, %1, 0x000f000f, %2, 0xEA;" : "=r"(a2) : "r"(w1), "r"(k1024));   // cols (2,6)
        asm("lop3.b32 %0, %1, 0x00f000f0, %2, 0xEA;" : "=r"(a3) : "r"(w1), "r"(k1024));   // cols (3,7) * 16
        o[4 * i + 0] = hmul2(hsub2(a0, k1032), s2);
        o[4 * i + 1] = hmul2(hsub2(a1, k1152), s2_16);
        o[4 * i + 2] = hmul2(hsub2(a2, k1032), s2);
        o[4 * i + 3] = hmul2(hsub2(a3, k1152), s2_16);
    }
}

// 32 columns of this lane -> 16: the sums with lane ^ 16, of columns 0..15 in the lower half of the warp, 16..31 in the upper.
__device__ __forceinline__ void sum_halves(const uint32_t (&v)[32], int upper, uint32_t (&o)[16]) {
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const float mine = __uint_as_float(upper ? v[16 + i] : v[i]), other = __uint_as_float(upper ? v[i] : v[16 + i]);
        o[i] = __float_as_uint(mine + __shfl_xor_sync(0xffffffffu, other, 16));
    }
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

// Mean of quantisation group g of a row as the correction chunks read it: chunk g / 32, K step (g % 32) / 8, columns
// g % 8 and 8 + g % 8 (against the hi and lo halves of the group's constant).
__device__ __forceinline__ void store_group_mean(__half* hi, __half* lo, size_t row, int g, float mean) {
    const __half h = __float2half_rn(mean), l = __float2half_rn(mean - __half2float(h));
    const size_t at = row + (size_t)(g >> 5) * TC_KC + ((g & 31) >> 3) * 16 + (g & 7);
    hi[at] = h; hi[at + 8] = h;
    lo[at] = l; lo[at + 8] = l;
}

// One unit of work: one token pass (up to 128 tokens) of one row tile of one expert group.
struct TcItem {
    int expert;   // local expert = slice of the weight maps
    int r0;       // first weight row of the tile (in each matrix)
    int grow;     // first grouped row of the pass
    int nt;       // tokens of the pass (1..128); 0 in a block's ring marks the end of the work
};

struct TcArgs {
    const TcItem* items;       // the launch's work list (written on the device)
    int* work;                 // [0] number of items, [1] next item to hand out, [2] most tokens of any item
    int R, C;                  // rows and columns of the weight matrices of this launch
    int extra;                 // split: correction chunks after a unit's C / 64 chunks
    __half* out_h;             // fused: GeGLU output [grouped rows][R] fp16, columns in operand K order
    __half* out_l;             // its fp16 residual (split precision) or null
    __half *sums_h, *sums_l;   // fused, split: group means of the GeGLU output in the correction chunks' K order
    int sums_stride;
    float* out_f;              // plain: projection output [grouped rows][R] fp32
    int* status;
    const uint32_t* tables;    // (scale << 16) | bias words, [local expert][3 tensors][C/64][R]: a chunk's words of 32 rows are one line
    const float* row_scale;    // split: power of two per weight row, [local expert][2 inter + hidden], gate | up | down ...
    const float* row_unscale;  // ... and its inverse
    int scale_stride;          // 2 inter + hidden
    int tensor0;               // first tensor of the slot this launch reads (0: gate, then up; 2: down)
    int scale_off;             // offset of that tensor's rows in row_scale (0, or 2 inter)
};

__device__ __forceinline__ uint32_t take_now(uint32_t v) {
    uint32_t r;
    asm volatile("mov.b32 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}
__device__ __forceinline__ uint32_t ldg_now(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// 32 bytes, 32-byte aligned, in one store.  The lanes of an epilogue warp write to 32 rows: every store instruction passes
// the L1 as 32 lines whatever its width, so a 16-byte one takes twice as long for the same bytes and leaves half sectors
// (a down unit of 128 tokens spent 4 to 8 us here with those).
__device__ __forceinline__ void store_sector(void* p, const uint32_t (&v)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
                 "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}

__device__ __forceinline__ uint4 lds_v4(const uint8_t* p) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(smem_u32(p)));
    return v;
}

// gelu_tanh(g) * u.  0.5 (1 + tanh i) = 1 / (1 + exp(-2 i)): a tenth of tanhf's instructions, and no cancellation for
// large negative g (the error of __expf grows with its argument: relative to the result a few 2^-23 near zero, |2 i| 2^-23 or
// so far from it, where the result is tiny; the epilogue of a unit of 44 chunks took 10000 cycles with tanhf).
__device__ __forceinline__ float geglu_fast(float g, float u) {
    const float inner = 0.7978845608028654f * (g + 0.044715f * g * g * g);
    return __fdividef(g * u, 1.0f + __expf(-2.0f * inner));
}

constexpr int TW_ROWS = 256;                        // rows of a converted stage
constexpr int TW_PK_BYTES = TW_ROWS * TC_KC / 2;    // packed chunk
constexpr int TW_B_BYTES = TW_ROWS * TC_KC * 2;     // converted chunk
constexpr int TW_TOK_BYTES = TC_MAX_NT * TC_KC * 2; // token tile of 128 rows
constexpr int TW_STAGES = 4;                        // most converted stages, and token tiles
constexpr int TW_PACK_MAX = 64;                     // split: passes of up to this many tokens carry hi and lo in ONE tile

template <bool FUSED, bool SPLIT>
__global__ void __launch_bounds__(TC_THREADS, 1)
q4_gemm_tc_kernel(const TcArgs a, const __grid_constant__ TcMaps maps, const __grid_constant__ TcMaps sums,
                  const __grid_constant__ TcWeightMaps wm) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bar_w[TC_MAX_SLOTS];     // packed chunk landed (TMA transaction bytes)
    __shared__ __align__(8) uint64_t bar_wfree[TC_MAX_SLOTS]; // ... and is in its converters' registers (8 warp arrivals)
    __shared__ __align__(8) uint64_t bar_tok[TW_STAGES];      // token tile landed
    __shared__ __align__(8) uint64_t bar_full[TW_STAGES];     // stage converted (8 warp arrivals)
    __shared__ __align__(8) uint64_t bar_done[TW_STAGES];     // the MMAs that read stage and token tile are complete
    // A unit = one token pass of one row tile.  Accumulators are double-buffered by unit parity (256 columns each).
    __shared__ __align__(8) uint64_t bar_acc[2];              // a unit's accumulators are final
    __shared__ __align__(8) uint64_t bar_epi[2];              // ... and have been read (16 warp arrivals)
    // The block draws units from the launch's work list (one atomic per unit, by the producing thread, which
    // passes the item to the other roles through a small ring).
    __shared__ __align__(16) TcItem s_items[TC_ITEM_RING];
    __shared__ __align__(8) uint64_t bar_item[TC_ITEM_RING];  // ring entry published
    __shared__ float s_half[2][TC_MAX_NT];                    // half sums of two 64-column groups (fused, split)
    __shared__ __align__(8) uint64_t bar_half[2][8];          // ... written by one warp of a pair, read by the other
    __shared__ uint32_t s_tmem;
    __shared__ int s_fail;

    constexpr int NMAT = FUSED ? 2 : 1;
    constexpr int RT = TW_ROWS / NMAT;                        // weight rows of a tile, per matrix
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nchunks = a.C / TC_KC, total = nchunks + (SPLIT ? a.extra : 0);
    // carve-up: converted stages | token tiles (room for the launch's largest pass) | packed chunks.  The MMA always
    // reads 128 token rows: those above the copied boxes are stale bytes and only reach accumulator lanes nobody reads.
    uint8_t* stage_base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int nt_max = *(volatile const int*)&a.work[2];
    const uint32_t tok_room = SPLIT ? (nt_max <= TW_PACK_MAX ? (uint32_t)TW_TOK_BYTES : 2u * TW_TOK_BYTES)
                                    : (nt_max <= 16 ? 2048u : nt_max <= 32 ? 4096u : nt_max <= 64 ? 8192u : (uint32_t)TW_TOK_BYTES);
    // stages, token tiles and packed chunks in flight: four of each (two stages per converter group), or three stages
    // where a token tile holds 128 rows of hi and of lo; the rest is packed chunks
    const uint32_t ND = tok_room <= (uint32_t)TW_TOK_BYTES ? 4u : 3u;
    uint8_t* tok_base = stage_base + ND * TW_B_BYTES;
    uint8_t* pk_base = tok_base + ND * tok_room;
    constexpr uint32_t NW = 4, nw_shift = 2;
    static_assert(TC_SMEM_BYTES - 1024 - 3 * (TW_B_BYTES + 2 * TW_TOK_BYTES) >= (int)NW * TW_PK_BYTES, "packed ring");
    static_assert(TC_SMEM_BYTES - 1024 - 4 * (TW_B_BYTES + TW_TOK_BYTES) >= (int)NW * TW_PK_BYTES, "packed ring");
    volatile int* fail = &s_fail;

    if (tid == 0) {
        for (int s = 0; s < TC_MAX_SLOTS; s++) {
            mbar_init(&bar_w[s], 1);
            mbar_init(&bar_wfree[s], TC_GROUP / 32);
        }
        for (int s = 0; s < TW_STAGES; s++) {
            mbar_init(&bar_tok[s], 1);
            mbar_init(&bar_full[s], TC_GROUP / 32);
            mbar_init(&bar_done[s], 1);
        }
        for (int s = 0; s < TC_ITEM_RING; s++) mbar_init(&bar_item[s], 1);
        for (int s = 0; s < 2; s++) {
            mbar_init(&bar_acc[s], 1);
            mbar_init(&bar_epi[s], TC_CONVERTERS / 32);
            for (int i = 0; i < 8; i++) mbar_init(&bar_half[s][i], 1);
        }
        s_fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                     "r"(TC_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    uint32_t requested = 0;       // copies requested by this thread / chunks committed (issuer)

    if (warp < TC_ISSUER_WARP) {
        // ================= converters, then the epilogue of every unit =================
        const uint32_t grp = (uint32_t)warp >> 3;
        const int crow = (warp & 7) * 32 + lane;                 // stage row
        uint8_t* const line = stage_base + (uint32_t)crow * 128; // the row's 128-byte line in the 256 x 64 fp16 tile
        const uint32_t b_sw = ((uint32_t)crow & 7) << 4;
        const NibbleMagic mg = load_nibble_magic();
        uint32_t it0 = 0, w0 = 0;                                // chunks, packed chunks before this unit
        uint32_t half_phase = 0;                                 // phase of this warp's half sums
        // Epilogue of a unit: warp w reads lane quarter w % 4 (tokens) and a quarter of the columns.
        auto epilogue = [&](const TcItem& item, uint32_t unit) -> bool {
            // the unit's row factors, a column per lane, on their way before the accumulators are final
            const int q = warp & 3, cq = warp >> 2, rows_here = min(RT, a.R - item.r0), r0 = item.r0;
            float un_a = 1.0f, un_b = 1.0f;                              // fused: gate, up; plain: columns 0..31, 32..63
            if (SPLIT) {
                const float* un = a.row_unscale + (size_t)item.expert * a.scale_stride + a.scale_off + r0;
                const int c = FUSED ? cq * 32 : cq * 64;
                if (c < rows_here) un_a = __ldg(un + c + lane);
                if (FUSED ? c < rows_here : c + 32 < rows_here) un_b = __ldg(un + (FUSED ? a.R + c : c + 32) + lane);
            }
            if (!__all_sync(0xffffffffu, mbar_wait(&bar_acc[unit & 1u], (unit >> 1) & 1u, fail))) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const bool packed = SPLIT && item.nt <= TW_PACK_MAX;
            // packed: lanes 0..15 of a quarter hold sixteen tokens' hi products, lanes 16..31 the lo products of the same
            // tokens; after their sum the two halves of the warp share the columns
            const int n = packed ? q * 16 + (lane & 15) : q * 32 + lane;         // token of the pass
            const int half0 = packed ? lane >> 4 : 0, halves = packed ? 1 : 2;
            const uint32_t trow = tmem + ((uint32_t)(q * 32) << 16) + (unit & 1u) * TW_ROWS;
            // sixteen columns of this lane: the sums of the two halves, or columns c ... c + 15
            auto sixteen = [&](uint32_t c, int h, uint32_t (&v)[16]) {
                if (packed) {
                    uint32_t t[32];
                    tmem_ld32(trow + c, t);
                    sum_halves(t, half0, v);
                } else {
                    tmem_ld16(trow + c + h * 16, v);
                }
            };
            if ((packed ? q * 16 : q * 32) < item.nt) {                          // warp-uniform: the quarter holds tokens
                if (FUSED) {
                    const int col = cq * 32;                                     // output columns col ... col + 31 of the tile
                    if (col < rows_here) {
                        float sum = 0.0f;
#pragma unroll 1
                        for (int h = 0; h < halves; h++) {
                            const int cc = (packed ? half0 : h) * 16, c0 = col + cc;
                            const size_t o_off = (size_t)(item.grow + n) * a.R + r0 + c0;
                            uint32_t g[16], u[16];
                            sixteen(col, h, g);
                            sixteen((rows_here > RT / 2 ? RT : RT / 2) + col, h, u);
                            float o[16];
#pragma unroll
                            for (int i = 0; i < 16; i++) {
                                float gv = __uint_as_float(g[i]), uv = __uint_as_float(u[i]);
                                if (SPLIT) {
                                    gv *= __shfl_sync(0xffffffffu, un_a, cc + i);
                                    uv *= __shfl_sync(0xffffffffu, un_b, cc + i);
                                }
                                o[i] = geglu_fast(gv, uv);
                                sum += o[i];
                            }
                            if (n < item.nt) {
                                // the next GEMM's K order inside a group of 8: [0,4,1,5,2,6,3,7]
                                uint32_t hw[8], lw[8];
#pragma unroll
                                for (int kk = 0; kk < 8; kk++) {
                                    const int i = (kk >> 2) * 8 + (kk & 3);
                                    hw[kk] = f16x2_from(o[i], o[i + 4]);
                                    if (SPLIT) lw[kk] = f16x2_from(o[i] - f16_lo_to_f32(hw[kk]), o[i + 4] - f16_hi_to_f32(hw[kk]));
                                }
                                store_sector(a.out_h + o_off, hw);
                                if (SPLIT) store_sector(a.out_l + o_off, lw);
                            }
                        }
                        if (SPLIT) {
                            // mean of a 64-column group: 32 columns here, 32 in the warp four further on
                            if (packed) sum += __shfl_xor_sync(0xffffffffu, sum, 16);
                            float* half = s_half[cq >> 1];
                            const int pair = q * 2 + (cq >> 1);
                            // the writer waits until the sums before have been read (at its first time: passes at once)
                            const uint32_t parity = half_phase ^ (uint32_t)(cq & 1);
                            half_phase ^= 1u;
                            if (!__all_sync(0xffffffffu, mbar_wait(&bar_half[cq & 1][pair], parity, fail))) return false;
                            if (cq & 1) {
                                half[n] = sum;
                            } else {
                                if (n < item.nt && (!packed || lane < 16))
                                    store_group_mean(a.sums_h, a.sums_l, (size_t)(item.grow + n) * a.sums_stride, (r0 + col) / TC_KC,
                                                     (sum + half[n]) * (1.0f / TC_KC));
                            }
                            __syncwarp();
                            if (lane == 0) mbar_arrive(&bar_half[(cq & 1) ^ 1][pair]);
                        }
                    }
                } else {
#pragma unroll 1
                    for (int c1 = 0; c1 < 64; c1 += 32) {
                        const int col = cq * 64 + c1;
                        if (col >= rows_here) break;
                        const float f = c1 ? un_b : un_a;
#pragma unroll 1
                        for (int h = 0; h < halves; h++) {
                            const int cc = (packed ? half0 : h) * 16;
                            uint32_t g[16];
                            sixteen(col, h, g);
                            float* dst = a.out_f + (size_t)(item.grow + n) * a.R + r0 + col + cc;
                            uint32_t o[2][8];
#pragma unroll
                            for (int i = 0; i < 16; i++)
                                o[i >> 3][i & 7] = SPLIT ? __float_as_uint(__uint_as_float(g[i]) * __shfl_sync(0xffffffffu, f, cc + i)) : g[i];
                            if (n < item.nt) {
                                store_sector(dst, o[0]);
                                store_sector(dst + 8, o[1]);
                            }
                        }
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar_epi[unit & 1u]);
            return true;
        };
        bool alive = true, pending = false;
        TcItem prev = {0, 0, 0, 0};
        for (uint32_t unit = 0; alive && !*fail; unit++) {
            alive = __all_sync(0xffffffffu, mbar_wait(&bar_item[unit % TC_ITEM_RING], (unit / TC_ITEM_RING) & 1u, fail));
            if (!alive) break;
            const TcItem item = s_items[unit % TC_ITEM_RING];
            const int mine = item.nt < 1 ? 0 : total;                    // nt < 1: end of the work
            // The last tile of gate and up may be 64 rows wide: the stage is then 64 rows of gate, 64 of up (one instruction of
            // half the width) and the other warps only keep step.
            const bool half = FUSED && a.R - item.r0 <= RT / 2;
            const int mat = FUSED ? (half ? crow / (RT / 2) & 1 : crow / RT) : 0;
            const int row = min(item.r0 + (half ? crow % (RT / 2) : crow % RT), a.R - 1);
            const uint32_t pk_off = half ? (uint32_t)(mat * RT + crow % (RT / 2)) * 32u : (uint32_t)crow * 32u;
            const uint32_t* tab = a.tables + (size_t)(item.expert * 3 + a.tensor0 + mat) * a.R * nchunks + row;     // + group * R
            float rs = 1.0f;
            if (SPLIT) rs = __ldg(a.row_scale + (size_t)item.expert * a.scale_stride + a.scale_off + mat * a.R + row);
            // this group's chunks of the unit: every other one of the block's running count
            const int first = (int)((it0 ^ grp) & 1u);
            uint32_t word_next = mine > 0 && first < nchunks ? __ldg(tab + (size_t)first * a.R) : 0u;
            // The unit before is finished after this group's second chunk: the tensor core has work while its accumulators
            // are read, and no converter waits for its last MMA.
            uint32_t w_here = 0u;
            for (int kc = first, n = 0;; kc += 2, n++) {
                if (pending && (n == 2 || kc >= mine)) {
                    pending = false;
                    if (!epilogue(prev, unit - 1)) { alive = false; break; }
                }
                if (kc >= mine) break;
                const uint32_t it = it0 + (uint32_t)kc, round = ND == 4u ? it >> 2 : it / 3u, s = it - round * ND;
                uint8_t* const st = line + s * TW_B_BYTES;
                if (FUSED && half && (warp & 4)) {
                    if (!SPLIT || kc < nchunks) {
                        const uint32_t slot = (w0 + kc) & (NW - 1), wph = ((w0 + kc) >> nw_shift) & 1u;
                        if (!__all_sync(0xffffffffu, mbar_wait(&bar_w[slot], wph, fail))) { alive = false; break; }
                        if (lane == 0) mbar_arrive(&bar_wfree[slot]);
                    }
                    if (round > 0 && !__all_sync(0xffffffffu, mbar_wait(&bar_done[s], (round - 1) & 1u, fail))) { alive = false; break; }
                } else if (!SPLIT || kc < nchunks) {
                    const uint32_t slot = (w0 + kc) & (NW - 1), wph = ((w0 + kc) >> nw_shift) & 1u;
                    // the next word a chunk pair ahead; this one is taken over BEFORE that load is issued, or waiting for it
                    // would also wait for the younger load on the same scoreboard (600 cycles a chunk)
                    const uint32_t word = take_now(word_next);
                    word_next = kc + 2 < nchunks ? ldg_now(tab + (size_t)(kc + 2) * a.R) : 0u;
                    if (!__all_sync(0xffffffffu, w_here) && !__all_sync(0xffffffffu, mbar_wait(&bar_w[slot], wph, fail))) { alive = false; break; }
                    const uint8_t* pk = pk_base + slot * TW_PK_BYTES + pk_off;
                    const uint4 p[2] = {lds_v4(pk), lds_v4(pk + 16)};
                    // the MMAs that last read this stage: asked now, needed after the conversion
                    uint32_t stage_free = round == 0 ? 1u : mbar_test(&bar_done[s], (round - 1) & 1u);
                    uint32_t o[2][16];
                    const uint32_t s_bits = word >> 16, b_bits = word & 0xffffu;
                    if (SPLIT) {
                        const float sc = bf16_bits_to_f32(s_bits) * rs;
                        const uint32_t s2 = f16x2_from(sc, sc), s2_16 = f16x2_from(sc * 0.0625f, sc * 0.0625f);
                        dequant_exact(p[0], s2, s2_16, o[0]);
                        dequant_exact(p[1], s2, s2_16, o[1]);
                    } else if (fp16_path_ok(s_bits, b_bits)) {
                        dequant_half_chunk_f16(p[0], s_bits, b_bits, o[0]);
                        dequant_half_chunk_f16(p[1], s_bits, b_bits, o[1]);
                    } else {
                        dequant_half_chunk_f32(mg, p[0], s_bits, b_bits, o[0]);
                        dequant_half_chunk_f32(mg, p[1], s_bits, b_bits, o[1]);
                    }
                    // this group's next packed chunk: asked now, needed in the next round (not across units: the slot's
                    // chunk before has to be one that this group has used, or the parity could be that of an older phase)
                    w_here = 0u;
                    if (kc + 2 < nchunks && kc + 2 >= (int)NW)
                        w_here = mbar_test(&bar_w[(w0 + kc + 2) & (NW - 1)], ((w0 + kc + 2) >> nw_shift) & 1u);
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bar_wfree[slot]);        // the packed bytes have been used
                    if (!__all_sync(0xffffffffu, stage_free) &&
                        !__all_sync(0xffffffffu, mbar_wait(&bar_done[s], (round - 1) & 1u, fail))) { alive = false; break; }
#pragma unroll
                    for (int i = 0; i < 8; i++)
                        *(uint4*)(st + (((uint32_t)i << 4) ^ b_sw)) =
                            make_uint4(o[i >> 2][4 * (i & 3)], o[i >> 2][4 * (i & 3) + 1], o[i >> 2][4 * (i & 3) + 2],
                                       o[i >> 2][4 * (i & 3) + 3]);
                } else {
                    // correction chunk: 32 groups, eight per K step of 16 columns: 64 c as hi, then as lo halves
                    const int g0 = (kc - nchunks) * 32;
                    uint32_t w[32];                                      // all words of the row at once: one latency
#pragma unroll
                    for (int j = 0; j < 32; j++) w[j] = g0 + j < nchunks ? ldg_now(tab + (size_t)(g0 + j) * a.R) : 0u;
                    if (round > 0 && !__all_sync(0xffffffffu, mbar_wait(&bar_done[s], (round - 1) & 1u, fail))) { alive = false; break; }
#pragma unroll
                    for (int ks = 0; ks < 4; ks++) {
                        uint32_t hi[4], lo[4];
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            float c[2];
#pragma unroll
                            for (int k = 0; k < 2; k++) {
                                const uint32_t v = w[ks * 8 + 2 * j + k];
                                c[k] = (bf16_bits_to_f32(v & 0xffffu) + 8.0f * bf16_bits_to_f32(v >> 16)) * (64.0f * rs);
                            }
                            hi[j] = f16x2_from(c[0], c[1]);
                            lo[j] = f16x2_from(c[0] - f16_lo_to_f32(hi[j]), c[1] - f16_hi_to_f32(hi[j]));
                        }
                        *(uint4*)(st + (((uint32_t)(2 * ks) << 4) ^ b_sw)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                        *(uint4*)(st + (((uint32_t)(2 * ks + 1) << 4) ^ b_sw)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
                    }
                }
                // generic-proxy writes -> visible to the tensor core (async proxy), then one arrival per warp
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar_full[s]);
            }
            if (mine == 0) break;
            it0 += (uint32_t)total;
            w0 += (uint32_t)nchunks;
            prev = item;
            pending = true;
        }
    } else if (warp == TC_ISSUER_WARP) {
        // ================= issuer (one thread) =================
        if (lane == 0) {
            const uint32_t w_lo0 = DESC_B_LO | ((smem_u32(stage_base) & 0x3ffffu) >> 4);
            const uint32_t t_lo0 = DESC_B_LO | ((smem_u32(tok_base) & 0x3ffffu) >> 4);
            uint32_t s = 0, ph = 0, ready = 0;
            bool ok = true;
            for (uint32_t unit = 0; ok && !*fail; unit++) {
                if (!mbar_wait(&bar_item[unit % TC_ITEM_RING], (unit / TC_ITEM_RING) & 1u, fail)) break;
                const TcItem item = s_items[unit % TC_ITEM_RING];
                if (item.nt < 1) break;                                  // end of the work
                const bool packed = item.nt <= TW_PACK_MAX;
                const uint32_t idesc = umma_idesc_f16(128, NMAT * min(RT, a.R - item.r0));
                // this unit's accumulator buffer was last used two units ago: those accumulators have been read
                if (unit >= 2 && !mbar_wait(&bar_epi[unit & 1u], ((unit >> 1) - 1) & 1u, fail)) { ok = false; break; }
                const uint32_t acc_base = tmem + (unit & 1u) * TW_ROWS;
                for (int kc = 0; kc < total; kc++) {
                    // the converted weights of the stage, and the chunk's token tile: the tensor core reads it
                    // through the async proxy, so the issuing thread observes that barrier itself
                    if (!ready) ok = mbar_wait2(&bar_full[s], ph, &bar_tok[s], ph, fail);
                    if (!ok) break;
                    // poll the next chunk's barriers now; the answer arrives behind this chunk's MMAs
                    const uint32_t ns = s + 1 == ND ? 0 : s + 1, nph = s + 1 == ND ? ph ^ 1u : ph;
                    const uint32_t r_full = mbar_test(&bar_full[ns], nph), r_tok = mbar_test(&bar_tok[ns], nph);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t wlo = w_lo0 + s * (TW_B_BYTES >> 4), tlo = t_lo0 + s * (tok_room >> 4);
#pragma unroll
                    for (int j = 0; j < TC_KC / 16; j++) {
                        const uint64_t w = make_desc(wlo + j * 2, DESC_B_HI);
                        umma_f16(acc_base, make_desc(tlo + j * 2, DESC_B_HI), w, idesc, (kc > 0 || j > 0) ? 1u : 0u);
                        if (SPLIT && !packed) umma_f16(acc_base, make_desc(tlo + (TW_TOK_BYTES >> 4) + j * 2, DESC_B_HI), w, idesc, 1u);
                    }
                    umma_commit(&bar_done[s]);
                    if (kc == total - 1) umma_commit(&bar_acc[unit & 1u]);
                    requested++;
                    ready = r_full & r_tok;
                    s = ns; ph = nph;
                }
            }
        }
    } else if (warp == TC_WEIGHT_WARP) {
        // ================= units and packed weights (one thread) =================
        if (lane == 0) {
            bool pok = true;
            const int n_items = *(volatile const int*)&a.work[0];
            for (uint32_t unit = 0; pok && !*fail; unit++) {
                const int idx = atomicAdd(&a.work[1], 1);
                TcItem item = {0, 0, 0, 0};
                if (idx < n_items) {
                    const int4 v = *(const int4*)&a.items[idx];
                    item.expert = v.x; item.r0 = v.y; item.grow = v.z; item.nt = v.w;
                }
                s_items[unit % TC_ITEM_RING] = item;
                mbar_arrive(&bar_item[unit % TC_ITEM_RING]);       // release: the entry is visible to who sees the phase
                if (item.nt < 1) break;
                for (int kc = 0; kc < nchunks; kc++) {
                    const uint32_t slot = requested & (NW - 1), round = requested >> nw_shift;
                    if (round > 0 && !mbar_wait(&bar_wfree[slot], (round - 1) & 1u, fail)) { pok = false; break; }
                    const uint32_t dst = smem_u32(pk_base + slot * TW_PK_BYTES);
                    mbar_expect_tx(&bar_w[slot], TW_PK_BYTES);
                    if (FUSED) {
                        // 128 rows of gate, then the same 128 rows of up
#pragma unroll
                        for (int m = 0; m < 2; m++)
                            tma_load_3d(dst + m * TC_PK_BYTES, &wm.w[m], kc * 32, item.r0, item.expert, &bar_w[slot]);
                    } else {
                        tma_load_3d(dst, &wm.w256, kc * 32, item.r0, item.expert, &bar_w[slot]);
                    }
                    requested++;
                }
            }
        }
    } else if (lane == 0) {
        // ================= token tiles (one thread) =================
        bool pok = true;
        for (uint32_t unit = 0; pok && !*fail; unit++) {
            if (!mbar_wait(&bar_item[unit % TC_ITEM_RING], (unit / TC_ITEM_RING) & 1u, fail)) break;
            const TcItem item = s_items[unit % TC_ITEM_RING];
            if (item.nt < 1) break;
            const bool packed = SPLIT && item.nt <= TW_PACK_MAX;
            const int boxes = (item.nt + 15) / 16;
            const int variant = item.nt <= 16 ? 0 : item.nt <= 32 ? 1 : item.nt <= 64 ? 2 : 3;
            const uint32_t bytes = packed ? (uint32_t)boxes * 2u * 2048u : (SPLIT ? 2u : 1u) * ((16u << variant) * 128u);
            for (int kc = 0; kc < total; kc++) {
                const uint32_t round = ND == 4u ? requested >> 2 : requested / 3u, s = requested - round * ND;
                if (round > 0 && !mbar_wait(&bar_done[s], (round - 1) & 1u, fail)) { pok = false; break; }
                const uint32_t dst = smem_u32(tok_base + s * tok_room);
                const TcMaps& m = kc < nchunks ? maps : sums;
                const int x = (kc < nchunks ? kc : kc - nchunks) * TC_KC;
                mbar_expect_tx(&bar_tok[s], bytes);
                if (packed) {
                    // sixteen tokens' hi rows, then their lo rows, in every quarter of the tile
                    for (int b = 0; b < boxes; b++) {
                        tma_load_2d(dst + b * 4096, &m.hi[0], x, item.grow + 16 * b, &bar_tok[s]);
                        tma_load_2d(dst + b * 4096 + 2048, &m.lo[0], x, item.grow + 16 * b, &bar_tok[s]);
                    }
                } else {
                    tma_load_2d(dst, &m.hi[variant], x, item.grow, &bar_tok[s]);
                    if (SPLIT) tma_load_2d(dst + TW_TOK_BYTES, &m.lo[variant], x, item.grow, &bar_tok[s]);
                }
                requested++;
            }
        }
    }
    if (*fail) {
        // wait (bounded, no early exit) for the copies and MMAs still in flight before shared memory and
        // TMEM are released
        int none = 0;
        if (lane == 0 && warp == TC_WEIGHT_WARP)
            for (uint32_t t = (requested > NW ? requested - NW : 0); t < requested; t++)
                (void)mbar_wait(&bar_w[t & (NW - 1)], (t >> nw_shift) & 1u, &none);
        if (lane == 0 && warp == TC_TOKEN_WARP)
            for (uint32_t t = (requested > ND ? requested - ND : 0); t < requested; t++)
                (void)mbar_wait(&bar_tok[t % ND], (t / ND) & 1u, &none);
        if (lane == 0 && warp == TC_ISSUER_WARP && requested > 0)
            (void)mbar_wait(&bar_done[(requested - 1) % ND], ((requested - 1) / ND) & 1u, &none);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (tid == 0 && *fail && a.status) atomicOr(a.status, SB_ERR_TIMEOUT);
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TC_TMEM_COLS) : "memory");
    }
}

// Work lists of a layer's two launches: for every expert group with tokens, every 128-token pass, every row
// tile one item (tiles of a pass adjacent, so neighbouring blocks share the pass' token rows in L2).  One block; a warp
// per group (all threads on one group after the other took 10 us for 128 groups).
struct WorkListArgs {
    const Q4Job* jobs;
    const int* njobs_dev;
    int njobs_max;
    const float* y_base;
    int y_cols;
    const uint8_t* pool;
    size_t expert_stride;
    int nx_fused, nx_plain;
    TcItem *items_fused, *items_plain;
    int* work;
};
__device__ __forceinline__ void write_work_lists(const WorkListArgs& a, int* s_list) {
    // s_list: [njobs_max + 1] first pass of every job, then expert, first row, tokens
    int* s_base = s_list;
    int* s_expert = s_list + a.njobs_max + 1;
    int* s_g0 = s_expert + a.njobs_max;
    int* s_ntok = s_g0 + a.njobs_max;
    const int njobs = a.njobs_dev ? min(*a.njobs_dev, a.njobs_max) : a.njobs_max;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int j = threadIdx.x; j < njobs; j += blockDim.x) {
        const Q4Job& jb = a.jobs[j];
        s_expert[j] = (int)((size_t)(jb.vals - a.pool) / a.expert_stride);
        s_g0[j] = (int)((jb.y - a.y_base) / a.y_cols);
        s_ntok[j] = max(jb.ntok, 0);
    }
    __syncthreads();
    if (warp == 0) {
        int run = 0, nt_max = 0;
        for (int j0 = 0; j0 < njobs; j0 += 32) {
            const int j = j0 + lane, ntok = j < njobs ? s_ntok[j] : 0, np = (ntok + TC_MAX_NT - 1) / TC_MAX_NT;
            int inc = np;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += t;
            }
            if (j < njobs) s_base[j] = run + inc - np;
            run += __shfl_sync(0xffffffffu, inc, 31);
            nt_max = max(nt_max, min(ntok, TC_MAX_NT));
        }
        nt_max = __reduce_max_sync(0xffffffffu, nt_max);
        if (lane == 0) {
            s_base[njobs] = run;
            a.work[0] = run * a.nx_fused; a.work[1] = 0; a.work[2] = nt_max;
            a.work[4] = run * a.nx_plain; a.work[5] = 0; a.work[6] = nt_max;
        }
    }
    __syncthreads();
    const int nxt = a.nx_fused + a.nx_plain;
    for (int j = warp; j < njobs; j += blockDim.x >> 5) {
        const int base = s_base[j], np = s_base[j + 1] - base;
        for (int p = 0; p < np; p++) {
            TcItem it;
            it.expert = s_expert[j]; it.grow = s_g0[j] + p * TC_MAX_NT; it.nt = min(TC_MAX_NT, s_ntok[j] - p * TC_MAX_NT);
            for (int x = lane; x < nxt; x += 32) {
                if (x < a.nx_fused) {
                    it.r0 = x * (TW_ROWS / 2);
                    a.items_fused[(size_t)(base + p) * a.nx_fused + x] = it;
                } else {
                    it.r0 = (x - a.nx_fused) * TW_ROWS;
                    a.items_plain[(size_t)(base + p) * a.nx_plain + (x - a.nx_fused)] = it;
                }
            }
        }
    }
}

// x (fp32, token rows) -> fp16 rows in grouped order: xh[c2g[t * topk + k]] = fp16(x[t]) for every selection k of token t,
// and (when xl != null) the residuals xl = fp16(x - xh) and the means of the 64-column groups.  Columns inside every group
// of 8 are written in the operands' K order.  A token's columns are loaded and converted once and stored topk times; with
// a block per GROUPED row (eight times the blocks, loads and conversions) and the work lists in a launch of their own, 69 us
// of a layer of 512 tokens and 99 of 1999 went into this and the first row-wise glue; now 37 and 46.
// blockIdx.y = 0: the work lists (one block), beside the rows: both need nothing but the plan.
constexpr int GATHER_THREADS = 128;
__global__ void __launch_bounds__(GATHER_THREADS)
scatter_convert_kernel(const float* __restrict__ x, const int32_t* __restrict__ c2g, __half* __restrict__ xh,
                       __half* __restrict__ xl, __half* __restrict__ sums_h, __half* __restrict__ sums_l, int sums_stride,
                       int jobs, int topk, int hidden, const WorkListArgs lists) {
    if (blockIdx.y == 0) {
        extern __shared__ int s_list[];
        if (blockIdx.x == 0) write_work_lists(lists, s_list);
        return;
    }
    const int token = blockIdx.y - 1;
    const int d = (blockIdx.x * GATHER_THREADS + threadIdx.x) * 8;
    if (d >= hidden) return;                      // hidden is a multiple of 64: the eight lanes of a group stay together
    const float* src = x + (size_t)token * hidden + d;
    const float4 v0 = *(const float4*)src, v1 = *(const float4*)(src + 4);
    const float v[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {   // half2 k holds columns (k, k + 4)
        hi[k] = f16x2_from(v[k], v[k + 4]);
        lo[k] = f16x2_from(v[k] - f16_lo_to_f32(hi[k]), v[k + 4] - f16_hi_to_f32(hi[k]));
    }
    float sum = 0.0f;
    if (xl) {
        sum = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
        const uint32_t octet = 0xffu << (threadIdx.x & 24);
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) sum += __shfl_xor_sync(octet, sum, o);
    }
#pragma unroll 4
    for (int k = 0; k < topk; k++) {
        const int g = __ldg(c2g + (size_t)token * topk + k);
        if (g < 0 || g >= jobs) continue;         // a selection without an expert (reported by the plan kernel)
        *(uint4*)(xh + (size_t)g * hidden + d) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        if (xl) {
            *(uint4*)(xl + (size_t)g * hidden + d) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            if ((threadIdx.x & 7) == 0) store_group_mean(sums_h, sums_l, (size_t)g * sums_stride, d / TC_KC, sum * (1.0f / TC_KC));
        }
    }
}

// Derived tables of an expert pool: the (scale << 16) | bias words by group instead of by row (a converter warp's 32 rows
// of a chunk lie in one line; by row its load touched 32 lines and took 300 to 500 cycles a chunk to issue), and
// powers of two that bring every weight row into fp16: the largest of 8 |s| and 64 |c| of a row becomes
// 2^9 .. 2^10.  Small scales of the row lose bits only below 2^-27 of its largest weight.
__global__ void __launch_bounds__(256)
q4_tc_tables_kernel(const uint32_t* __restrict__ tables, int hidden, int inter, int experts, uint32_t* __restrict__ by_group,
                    float* __restrict__ scale, float* __restrict__ unscale) {
    const int per = 2 * inter + hidden, n = experts * per;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int e = i / per, r = i % per, k = r < inter ? 0 : (r < 2 * inter ? 1 : 2), row = r - k * inter;
        const int groups = (k < 2 ? hidden : inter) / TC_KC;
        const size_t tensor = (size_t)(e * 3 + k) * ((size_t)hidden * inter / TC_KC);
        const uint32_t* t = tables + tensor + (size_t)row * groups;
        uint32_t* o = by_group + tensor + row;
        const int rows = k < 2 ? inter : hidden;
        float top = 0.0f;
        for (int g = 0; g < groups; g++) {
            const float s = bf16_bits_to_f32(t[g] >> 16), b = bf16_bits_to_f32(t[g] & 0xffffu);
            top = fmaxf(top, fmaxf(8.0f * fabsf(s), 64.0f * fabsf(b + 8.0f * s)));
            o[(size_t)g * rows] = t[g];
        }
        int ex = 0;
        if (top > 0.0f && top < 3.0e38f) frexpf(top, &ex);       // top = m 2^ex, 1/2 <= m < 1
        ex = min(max(10 - ex, -100), 100);
        scale[i] = ldexpf(1.0f, ex);
        unscale[i] = ldexpf(1.0f, -ex);
    }
}

cudaError_t launch_q4_tc_tables(const uint32_t* tables, int hidden, int inter, int experts, uint32_t* by_group, float* scale,
                                float* unscale, cudaStream_t stream) {
    if (experts < 1) return cudaSuccess;
    q4_tc_tables_kernel<<<592, 256, 0, stream>>>(tables, hidden, inter, experts, by_group, scale, unscale);
    return launched();
}

cudaError_t tensor_map_encoder(TensorMapEncodeFn* out) {
    static TensorMapEncodeFn encode = nullptr;     // the entry point is process-wide, not per device
    if (!encode) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
        if (e != cudaSuccess) return e;
        if (!fn || q != cudaDriverEntryPointSuccess) return cudaErrorNotSupported;
        encode = (TensorMapEncodeFn)fn;
    }
    *out = encode;
    return cudaSuccess;
}

// Tensor maps over a [rows][cols] fp16 buffer (and its residual buffer): boxes of 64
// columns x 16 / 32 / 64 / 128 rows, 128-byte swizzle, zero fill past the last row.
cudaError_t make_tc_maps(TcMaps* out, const void* hi, const void* lo, int rows, int cols) {
    TensorMapEncodeFn encode = nullptr;
    {
        cudaError_t e = tensor_map_encoder(&encode);
        if (e != cudaSuccess) return e;
    }
    if ((cols % TC_KC) != 0 || rows < 1) return cudaErrorInvalidValue;
    for (int v = 0; v < 4; v++)
        for (int part = 0; part < 2; part++) {
            const void* base = part ? lo : hi;
            if (!base) return cudaErrorInvalidValue;
            cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
            cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
            cuuint32_t box[2] = {(cuuint32_t)TC_KC, (cuuint32_t)(16 << v)};
            cuuint32_t estr[2] = {1, 1};
            CUresult r = encode(part ? &out->lo[v] : &out->hi[v], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
                                const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
            if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;
        }
    return cudaSuccess;
}

// Tiled maps over a layer's expert pool: packed nibbles as [C/2 bytes][R rows][experts] in boxes of one chunk (32 bytes) x
// 128 rows of gate and of up, 256 rows of down.  Rows past R read as zero.
cudaError_t make_q4_tc_weight_maps(TcWeightMaps* out, const uint8_t* pool, size_t expert_stride, const uint32_t* tables,
                                   const float* row_scale, const float* row_unscale, int hidden, int inter, int experts) {
    TensorMapEncodeFn encode = nullptr;
    {
        cudaError_t e = tensor_map_encoder(&encode);
        if (e != cudaSuccess) return e;
    }
    if ((hidden % TC_KC) != 0 || (inter % TC_KC) != 0 || experts < 1 || (expert_stride % 16) != 0 ||
        ((uintptr_t)pool % 16) != 0 || tables == nullptr || row_scale == nullptr || row_unscale == nullptr)
        return cudaErrorInvalidValue;
    const size_t elems = (size_t)hidden * inter;
    const size_t tensor_bytes = elems / 2 + 2 * (elems / 64 * 2);
    if ((tensor_bytes % 16) != 0) return cudaErrorInvalidValue;
    for (int k = 0; k < 3; k++) {
        const int R = k < 2 ? inter : hidden, C = k < 2 ? hidden : inter;
        cuuint64_t dims[3] = {(cuuint64_t)(C / 2), (cuuint64_t)R, (cuuint64_t)experts};
        cuuint64_t strides[2] = {(cuuint64_t)(C / 2), (cuuint64_t)expert_stride};
        cuuint32_t box[3] = {(cuuint32_t)(TC_KC / 2), k < 2 ? 128u : (cuuint32_t)TW_ROWS, 1u};
        cuuint32_t estr[3] = {1, 1, 1};
        CUresult r = encode(k < 2 ? &out->w[k] : &out->w256, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3,
                            const_cast<uint8_t*>(pool + (size_t)k * tensor_bytes), dims, strides, box, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;
    }
    out->pool = pool;
    out->expert_stride = expert_stride;
    out->tables = tables;
    out->row_scale = row_scale;
    out->row_unscale = row_unscale;
    return cudaSuccess;
}

// The limits of the two precisions are those the calls have always documented.  They come from tables that an earlier form
// kept in shared memory for sizes that are no multiple of 256; nothing in this form needs them, and nothing was tested beyond.
bool q4_tc_supported(int hidden, int inter, bool split) {
    if (hidden < TC_KC || inter < TC_KC || (hidden % TC_KC) || (inter % TC_KC)) return false;
    const int limit = split ? 960 : 3520;
    return ((hidden % 256) == 0 || hidden <= limit) && ((inter % 256) == 0 || inter <= limit);
}

template <bool FUSED, bool SPLIT>
static cudaError_t launch_tc(const TcArgs& a, const TcMaps& maps, const TcMaps& sums, const TcWeightMaps& wm, dim3 grid,
                             cudaStream_t stream) {
    {
        cudaError_t e = ensure_dynamic_smem((const void*)q4_gemm_tc_kernel<FUSED, SPLIT>, (size_t)TC_SMEM_BYTES);
        if (e != cudaSuccess) return e;
    }
    q4_gemm_tc_kernel<FUSED, SPLIT><<<grid, TC_THREADS, TC_SMEM_BYTES, stream>>>(a, maps, sums, wm);
    return launched();
}

size_t q4_tc_work_items_max(int n_experts, int rows_total, int hidden, int inter) {
    const size_t passes = (size_t)n_experts + (size_t)rows_total / TC_MAX_NT + 1;
    return passes * (size_t)std::max((inter + 127) / 128, (hidden + TW_ROWS - 1) / TW_ROWS);
}

cudaError_t launch_tc_prepare(const float* x, const int32_t* c2g, void* xh, void* xl, void* sums_h, void* sums_l, int rows,
                              int topk, int hidden, int inter, const Q4Job* gateup_jobs, const int* njobs_dev, int njobs_max,
                              const float* y_base, int y_cols, const TcWeightMaps& wm, void* items_fused, void* items_plain,
                              int* work, cudaStream_t stream) {
    if (rows < 1 || njobs_max < 1) return cudaSuccess;
    if (hidden % 64 || rows >= 65535) return cudaErrorInvalidValue;
    const WorkListArgs lists = {gateup_jobs, njobs_dev, njobs_max, y_base, y_cols, wm.pool, wm.expert_stride, (inter + 127) / 128,
                                (hidden + TW_ROWS - 1) / TW_ROWS, (TcItem*)items_fused, (TcItem*)items_plain, work};
    const dim3 grid((hidden / 8 + GATHER_THREADS - 1) / GATHER_THREADS, rows + 1);
    scatter_convert_kernel<<<grid, GATHER_THREADS, (size_t)(4 * njobs_max + 1) * sizeof(int), stream>>>(
        x, c2g, (__half*)xh, (__half*)xl, (__half*)sums_h, (__half*)sums_l, tc_sums_cols(hidden), rows * topk, topk, hidden, lists);
    return launched();
}

cudaError_t launch_q4_gemm_tc(bool fused, bool split, const void* items, int* work, const TcMaps& x, const TcMaps& sums,
                              const TcWeightMaps& wm, void* out_h, void* out_l, void* sums_h, void* sums_l, float* out_f, int R,
                              int C, int* status, cudaStream_t stream) {
    TcArgs a;
    a.items = (const TcItem*)items; a.work = work;
    a.R = R; a.C = C;
    a.extra = tc_sums_cols(C) / TC_KC;
    a.out_h = (__half*)out_h; a.out_l = (__half*)out_l; a.out_f = out_f; a.status = status;
    a.sums_h = (__half*)sums_h; a.sums_l = (__half*)sums_l; a.sums_stride = tc_sums_cols(R);
    a.tables = wm.tables;
    a.tensor0 = fused ? 0 : 2;
    a.row_scale = wm.row_scale; a.row_unscale = wm.row_unscale;
    const int inter = fused ? R : C, hidden = fused ? C : R;
    a.scale_stride = 2 * inter + hidden;
    a.scale_off = fused ? 0 : 2 * inter;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    // one resident block per SM; each draws units (one token pass of one row tile) from the work list until it is empty
    dim3 grid((unsigned)sms, 1, 1);
    if (fused)
        return split ? launch_tc<true, true>(a, x, sums, wm, grid, stream) : launch_tc<true, false>(a, x, sums, wm, grid, stream);
    return split ? launch_tc<false, true>(a, x, sums, wm, grid, stream) : launch_tc<false, false>(a, x, sums, wm, grid, stream);
}

}  // namespace sb
