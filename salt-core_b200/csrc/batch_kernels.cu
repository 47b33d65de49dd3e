// Affine-Q4 and NVFP4 projections of jobs of any number of tokens, exact (the reference row DAG of q4_core.cuh; NVFP4:
// reference src/nvfp4.c:157-192, the same 32 accumulators over dequantised activations).
//
// What bounds this work is not HBM: a weight element costs one product and one add per token (the reference
// rounds between them, so they cannot fuse), and at decode batches the activations that feed those two
// operations come out of shared memory.  A 32-lane shared load moves 4 bytes per lane and SM cycle, so with two
// weight rows and two columns per lane the activation loads alone took as long as the arithmetic.  Here a lane
// keeps RL = 4 rows (2 where the blocks would be few): eight lanes share a row (lane u owns accumulators 4u .. 4u + 3,
// two packed bytes of every 32-column step) and a 16-byte activation load feeds sixteen products.
//
//   * K is walked in chunks of 256 columns through a ring of shared-memory stages (128 bytes of every weight
//     row, and the activations of the tokens of the pass), filled by 16-byte cp.async; the weight rows of a stage
//     are 128 bytes apart and their 16-byte pieces are permuted by the row index, so the four rows a warp reads
//     together never share a bank.
//   * Q4: (scale << 16) | bias words of all rows of the tile are interleaved once per tile.  NVFP4: the block scales
//     of a chunk travel with it and index the 256 products fl(E4M3 code * global scale).
//   * A block takes up to four tokens of the group (its pass), with code specialised for 1, 2, 3 and 4; the passes of
//     a large group are blocks of their own, so that popular experts do not finish last.
//   * Dequantisation: a nibble masked at bits 16..19 (12..15) and OR-ed with the exponent of 2^7 (2^11) IS the
//     float 2^7 + q (2^11 + q), and d = fl(q*s + b) = fma(2^k + q, s, b - 2^k s) whenever b - 2^k s is exact,
//     which the tile checks for all of its groups; tiles with a group where it may not be take the two-rounding form.
//     (A group of equal weights whose quantiser keeps a least scale is one.)
//   * The canonical fold goes through a shared-memory area of the warp, two lanes per row, and the GeGLU of the
//     pass' tokens is spread over the lanes, instead of running on one lane in sixteen.
//
// What bounds it now: issue cycles.  Per row, lane and 32-column step a token takes four packed operations, each of which
// holds a scheduler for two cycles.  At 64 tokens (gate/up) 63 of 193 M warp instructions are these: 43 % of the launch's
// cycles; the others (dequantisation once per pass and row, activation loads, the blocks' tables, prologues and folds) are
// another 44 %.  At 16 tokens, where nearly every pass holds one or two, the products are 16 of 65 M.  Measured
// (hidden 2816, inter 704, 128 experts, top-8; gate/up + down of a layer, event pairs): 64 tokens 698 -> 409 us, 16 tokens
// 274 -> 150 us, 6 tokens 140 -> 87 us against two rows per lane and whole groups as blocks; 2 tokens 44 us, where one
// persistent launch for both phases took 51.
// NVFP4 (hidden 5120, inter 1536, 64 experts, top-4; expert phase of a layer): 1 token 71 -> 51 us, 16 tokens 640 -> 291; whole
// layers with jobs of passes instead of empty blocks: 16 tokens 338 -> 305 us, 64 tokens 867 -> 766, 256 tokens 3020 -> 2570.
#include "fp4_core.cuh"
#include "internal.h"
#include "pdl.cuh"
#include "q4_core.cuh"

namespace sb {
namespace {

// Exponent pattern of 2^7 (see c_nibble_magic: in a register, mask-and-or is one logic operation).
__constant__ uint32_t c_magic_2_7 = 0x43000000u;

constexpr int CH_COLS = 256;                // columns of a chunk
constexpr int CH_STEPS = CH_COLS / 32;      // 32-column steps of a chunk
constexpr int CH_BYTES = CH_COLS / 2;       // packed bytes per row and chunk
constexpr int STAGES = 3;                   // ring depth
constexpr int MAX_T = Q4_PASS_TOKENS;       // tokens per pass
constexpr int FOLD_BYTES = 4 * 8 * 16;       // fold area of a warp's four rows: eight float4 each
constexpr int WARPS = 4, NT = 32 * WARPS;

enum { FMT_Q4 = 0, FMT_FP4 = 1 };
enum { STEP_Q4 = 0, STEP_Q4_LITERAL = 1, STEP_FP4 = 2 };   // dequantisation of the inner loop

// Shared memory of a block: ring of stages | fold areas (one per warp) | table.  Stage: 128 bytes of every weight row,
// 256 columns of every token and, for NVFP4, 16 block scales of every row.  Table: (scale << 16) | bias words of the
// rows, or the 256 products fl(E4M3 code * global scale).  The raw Q4 scales and biases land where the last stage and
// the fold areas will be; they are gone before either is used.
struct BatchGeom {
    int rows, tpitch, raw_pitch, raw_block;
    uint32_t x_off, sc_off, stage_bytes, fold_off, table_off, raw_off, smem;
};
__host__ __device__ inline BatchGeom batch_geom(int fmt, int C, int nmat, int rl) {
    BatchGeom g;
    g.rows = WARPS * 4 * rl;
    g.tpitch = (C >> 6) + ((C >> 6) % 16 == 0 ? 1 : 0);   // the four rows a warp reads together fall in different banks
    g.raw_pitch = C >> 5;                   // bytes of bf16 scales per row
    g.raw_block = (g.rows / nmat * g.raw_pitch + 15) & ~15;
    g.x_off = (uint32_t)(g.rows * CH_BYTES);
    g.sc_off = g.x_off + MAX_T * CH_COLS * 4;
    g.stage_bytes = g.sc_off + (fmt == FMT_FP4 ? (uint32_t)g.rows * 16 : 0u);
    g.fold_off = g.stage_bytes * STAGES;
    g.raw_off = g.stage_bytes * (STAGES - 1);
    const uint32_t fold_end = g.fold_off + (uint32_t)(WARPS * rl * FOLD_BYTES);
    const uint32_t raw_end = fmt == FMT_FP4 ? 0u : g.raw_off + (uint32_t)(2 * nmat * g.raw_block);
    g.table_off = fold_end > raw_end ? fold_end : raw_end;
    const uint32_t table = fmt == FMT_FP4 ? 1024u : (uint32_t)(g.rows * g.tpitch * 4);
    const uint32_t out = (uint32_t)(MAX_T * g.rows * 4);    // the results of a block pass through the table's space
    g.smem = g.table_off + (table > out ? table : out);
    return g;
}

// May a group with these bf16 scale and bias bits be dequantised with one rounding, i.e. are b - 2^11 s and b - 2^7 s exact?
// Both have 8-bit significands, so a difference spans at most |exponent of b - exponent of 2^k s| + 9 bits and fits the 24
// of a float while 2^-4 |s| <= |b| < 2^22 |s| (by exponents); it is exact too if either is zero.  The bound on the scale
// keeps everything finite.  (Forming the difference, adding 2^k s back and comparing with b does not do: an error of half a
// unit of b's last place disappears in that sum.)  The usual groups need only near_key <= NEAR_MAX, which a tile tests as one
// maximum: zeros are looked at when that fails.  The exact error by a two-sum, or all of this for every group, cost up to 3 %
// of a layer of 16 to 64 tokens.
constexpr uint32_t NEAR_MAX = 26u << 7, SCALE_MAX = 230u << 7;
__device__ __forceinline__ uint32_t near_key(uint32_t hs, uint32_t hb) { return (hb & 0x7f80u) - (hs & 0x7f80u) + (4u << 7); }
__device__ __forceinline__ bool one_rounding(uint32_t hs, uint32_t hb) {
    if ((hs & 0x7fffu) == 0u) return true;
    return (hs & 0x7f80u) <= SCALE_MAX && (near_key(hs, hb) <= NEAR_MAX || (hb & 0x7fffu) == 0u);
}

// Two bytes (columns 4u .. 4u + 3) of one row as weights.  Scalar on purpose: a packed operation takes two issue
// cycles like two scalar ones, and pairs of equal scales would have to be moved into place first.
template <bool LIT>
__device__ __forceinline__ void dequant4(uint32_t h, float s, float c11, float c7, uint32_t m11, uint32_t m7, f32x2& d01, f32x2& d23) {
    const uint32_t b0 = h << 12, b1 = h << 4;
    float q[4];
    asm("lop3.b32 %0, %1, 0xf000, %2, 0xEA;" : "=f"(q[0]) : "r"(b0), "r"(m11));
    asm("lop3.b32 %0, %1, 0xf0000, %2, 0xEA;" : "=f"(q[1]) : "r"(b0), "r"(m7));
    asm("lop3.b32 %0, %1, 0xf000, %2, 0xEA;" : "=f"(q[2]) : "r"(b1), "r"(m11));
    asm("lop3.b32 %0, %1, 0xf0000, %2, 0xEA;" : "=f"(q[3]) : "r"(b1), "r"(m7));
    if (LIT) {          // c11 = c7 = b: fl(fl(q * s) + b), two roundings
#pragma unroll
        for (int i = 0; i < 4; i++) q[i] = __fadd_rn(__fmul_rn(__fadd_rn(q[i], i & 1 ? -128.0f : -2048.0f), s), c7);
    } else {            // c11 = b - 2^11 s, c7 = b - 2^7 s, both exact
#pragma unroll
        for (int i = 0; i < 4; i++) q[i] = __fmaf_rn(q[i], s, i & 1 ? c7 : c11);
    }
    d01 = pack2(q[0], q[1]);
    d23 = pack2(q[2], q[3]);
}

// One quantisation group (two 32-column steps) for RL rows and T tokens.
//   w: this lane's two bytes of step 0 at offset o0, of step 1 at o1, row i at + i * ISTEP * CH_BYTES
template <int RL, int T, bool LIT>
__device__ __forceinline__ void group_step(const uint8_t* w, uint32_t o0, uint32_t o1, const uint32_t* tab, int tab_row,
                                           const float* x, f32x2 (&acc)[RL][T][2], uint32_t m11, uint32_t m7, f32x2 nz) {
    constexpr int ISTEP = RL == 4 ? 8 : 16;
    float s[RL], c11[RL], c7[RL];
#pragma unroll
    for (int i = 0; i < RL; i++) {
        const uint32_t word = tab[i * tab_row];
        const float b = __uint_as_float(word << 16);
        s[i] = __uint_as_float(word & 0xffff0000u);
        c11[i] = LIT ? b : __fmaf_rn(-2048.0f, s[i], b);
        c7[i] = LIT ? b : __fmaf_rn(-128.0f, s[i], b);
    }
#pragma unroll
    for (int half = 0; half < 2; half++) {
        f32x2 x01[T], x23[T];
#pragma unroll
        for (int t = 0; t < T; t++) {
            const ulonglong2 xv = *(const ulonglong2*)(x + t * CH_COLS + half * 32);
            x01[t] = xv.x;
            x23[t] = xv.y;
        }
#pragma unroll
        for (int i = 0; i < RL; i++) {
            const uint32_t h = *(const uint16_t*)(w + (half ? o1 : o0) + i * ISTEP * CH_BYTES);
            f32x2 d01, d23;
            dequant4<LIT>(h, s[i], c11[i], c7[i], m11, m7, d01, d23);
#pragma unroll
            for (int t = 0; t < T; t++) {
                product_then_add(acc[i][t][0], d01, x01[t], nz);
                product_then_add(acc[i][t][1], d23, x23[t], nz);
            }
        }
    }
}

// Two 32-column steps of NVFP4 rows: w = fl(code * fl(scale * global)), one scale per 16 columns.  The hardware decodes
// the code 8 as -0 where the reference's table has +0 (src/nvfp4.c:19-23): as a weight that cannot change a result (the
// product is a zero of either sign, and an accumulator that starts at +0 never becomes -0).
template <int RL, int T>
__device__ __forceinline__ void group_step_fp4(const uint8_t* w, uint32_t o0, uint32_t o1, const uint8_t* sc, const float* lut,
                                               const float* x, f32x2 (&acc)[RL][T][2], f32x2 nz) {
    constexpr int ISTEP = RL == 4 ? 8 : 16;
#pragma unroll
    for (int half = 0; half < 2; half++) {
        f32x2 x01[T], x23[T];
#pragma unroll
        for (int t = 0; t < T; t++) {
            const ulonglong2 xv = *(const ulonglong2*)(x + t * CH_COLS + half * 32);
            x01[t] = xv.x;
            x23[t] = xv.y;
        }
#pragma unroll
        for (int i = 0; i < RL; i++) {
            const uint32_t h = *(const uint16_t*)(w + (half ? o1 : o0) + i * ISTEP * CH_BYTES);
            const float s = lut[sc[i * ISTEP * 16 + 2 * half]];
            float c[4];
            e2m1x4(h, c);
            const f32x2 d01 = pack2(__fmul_rn(c[0], s), __fmul_rn(c[1], s)), d23 = pack2(__fmul_rn(c[2], s), __fmul_rn(c[3], s));
#pragma unroll
            for (int t = 0; t < T; t++) {
                product_then_add(acc[i][t][0], d01, x01[t], nz);
                product_then_add(acc[i][t][1], d23, x23[t], nz);
            }
        }
    }
}

// The lane's global row of shared row `sr` (NMAT == 2: sixteen gate rows, then the same sixteen up rows, and so on).
template <int NMAT>
__device__ __forceinline__ int tile_row(int sr) {
    return NMAT == 2 ? (sr >> 5) * 16 + (sr & 15) : sr;
}

// Fold and store one pass of T tokens.  acc[i]: shared row sr0 + ISTEP i, tokens t.
template <int NMAT, int RL, int T>
__device__ __forceinline__ void finish_pass(const Q4Job& jb, int r0, int nvalid, int tb, float4* fold, float* out,
                                            int sr0, const f32x2 (&acc)[RL][T][2]) {
    constexpr int LPR = 8 / RL, ISTEP = RL == 4 ? 8 : 16;    // lanes per row of the warp
    static_assert(RL == 2 || RL == 4, "half of a lane's rows are gate rows, the others the up rows of the same outputs");
    const int lane = threadIdx.x & 31, u = lane & 7, lrow = lane >> 3;
    const int rr = lane / LPR, par = lane % LPR;             // this lane runs chain par and, with two lanes, par + 2
    float y[T];
#pragma unroll
    for (int t = 0; t < T; t++) {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < RL; i++) {
            float4 q;
            unpack2(acc[i][t][0], q.x, q.y);
            unpack2(acc[i][t][1], q.z, q.w);
            fold[(i * 4 + lrow) * 8 + (u ^ ((i * 4 + lrow) & 7))] = q;
        }
        __syncwarp();
        const float* a = (const float*)(fold + rr * 8) + par;
        float la = 0.0f, lb = 0.0f;                         // L_par, L_(par + 2)
#pragma unroll
        for (int s = 0; s < 8; s++) {
            la = __fadd_rn(la, a[4 * (s ^ (rr & 7))]);
            if (LPR == 2) lb = __fadd_rn(lb, a[4 * (s ^ (rr & 7)) + 2]);
        }
        if (LPR == 4) lb = __shfl_xor_sync(0xffffffffu, la, 2);
        const float mine = __fadd_rn(la, lb);
        y[t] = __fadd_rn(mine, __shfl_xor_sync(0xffffffffu, mine, 1));   // (L0 + L2) + (L1 + L3)
    }
    // row rr of the warp is shared row sr_w + ISTEP (rr >> 2) + (rr & 3)
    const int sr_w = sr0 - lrow;
    if (NMAT == 2) {
        // lanes 0..15 hold gate rows, lanes 16..31 the up rows of the same outputs; the tokens are spread over the
        // lanes of a row (and, with two lanes per row, over the halves), so that all share one evaluation of the GeGLU
        float gate = 0.0f, up = 0.0f;
        const int tok = LPR == 2 ? (lane >> 4) * 2 + par : par;
#pragma unroll
        for (int t = 0; t < T; t++) {
            const float other = __shfl_xor_sync(0xffffffffu, y[t], 16);
            if (t == tok) {
                gate = lane < 16 ? y[t] : other;
                up = lane < 16 ? other : y[t];
            }
        }
        const int g = rr & (2 * RL - 1);
        const int row = tile_row<2>(sr_w + ISTEP * (g >> 2) + (g & 3));
        if (tok < T && row < nvalid && (LPR == 2 || lane < 16))
            jb.y[(size_t)(tb + tok) * jb.y_stride + r0 + row] = __fmul_rn(gelu_tanh_exact(gate), up);
    } else {
        // through the (now unused) table, so that whole lines leave the block: the rows may be in host memory
        constexpr int ROWS = WARPS * 4 * RL;
        const int row = sr_w + ISTEP * (rr >> 2) + (rr & 3);
        __syncthreads();
#pragma unroll
        for (int t = 0; t < T; t++)
            if (t % LPR == par) out[t * ROWS + row] = y[t];
        __syncthreads();
        for (int i = threadIdx.x; i < T * ROWS; i += NT)
            if (i % ROWS < nvalid) jb.y[(size_t)(tb + i / ROWS) * jb.y_stride + r0 + i % ROWS] = out[i];
    }
}

// The stream of chunks of a block, 256 columns at a time.  A stage holds 16-byte pieces: eight per weight row (thread t
// copies piece t & 7 of rows (t >> 3) + k NT / 8, k = 0..RL - 1; gate rows for even k and up rows for odd k, or one
// matrix) and 64 per token.
template <int NMAT, int RL>
struct Loader {
    static constexpr int RSTEP = NT / 8, ROWS = WARPS * 4 * RL;
    static_assert(RSTEP == 16 && ROWS % 16 == 0, "even k = gate rows, odd k = up rows");
    const Q4Job& jb;                 // in shared memory, as are the activation rows: registers are what is short
    const float* const* rows;        // [ntok]
    const uint8_t* src;              // this thread's piece of chunk 0 in its first row
    int r0, below, ch, ntok, steps;  // first row of the tile; rows below this thread's first one; next chunk

    __device__ __forceinline__ Loader(const Q4Job& j, const float* const* rows_, int r0_, int C, int ntok_)
        : jb(j), rows(rows_), r0(r0_), ch(0), ntok(ntok_), steps(C >> 5) {
        const int row = min(r0 + (int)(threadIdx.x >> 3), jb.R - 1);
        below = jb.R - 1 - row;
        src = jb.vals + (size_t)row * (C >> 1) + (threadIdx.x & 7) * 16;
    }
    __device__ __forceinline__ bool more() const { return ch * CH_STEPS < steps; }
    __device__ __forceinline__ void weights(uint8_t* stage) const {
        const int pc = threadIdx.x & 7, sr = threadIdx.x >> 3;
        if (pc >= steps - ch * CH_STEPS) return;
        uint8_t* dst = stage + sr * CH_BYTES + ((pc ^ (sr & 7)) << 4);   // RSTEP is a multiple of 8: the same permutation for all k
        const uint8_t* p = src + ch * CH_BYTES;
        const ptrdiff_t second = NMAT == 2 ? jb.vals2 - jb.vals : 0;
#pragma unroll
        for (int k = 0; k < RL; k++) {
            const int down = min(NMAT == 2 ? (k >> 1) * RSTEP : k * RSTEP, below);
            cp_async16(dst + k * RSTEP * CH_BYTES, p + (size_t)(down * steps) * 16 + (NMAT == 2 && (k & 1) ? second : 0));
        }
    }
    __device__ __forceinline__ void block_scales(uint8_t* stage) const {    // NVFP4: 16 per row and chunk
        if (threadIdx.x < ROWS) {
            const int row = min(r0 + (int)threadIdx.x, jb.R - 1);
            cp_async16(stage + threadIdx.x * 16, jb.scales + (size_t)row * (steps * 2) + ch * 16);
        }
    }
    __device__ __forceinline__ void activations(uint8_t* stage) const {
#pragma unroll
        for (int k = 0; k < (MAX_T * 64 + NT - 1) / NT; k++) {
            const int idx = threadIdx.x + k * NT, t = idx >> 6, pc = idx & 63;
            if (t < ntok && pc < (steps - ch * CH_STEPS) * 8)
                cp_async16(stage + idx * 16, rows[t] + ch * CH_COLS + pc * 4);
        }
    }
};

template <int FMT, int NMAT, int RL>
__device__ __forceinline__ void load_chunk(Loader<NMAT, RL>& ld, const BatchGeom& G, uint8_t* stage) {
    if (ld.more()) {
        ld.weights(stage);
        ld.activations(stage + G.x_off);
        if (FMT == FMT_FP4) ld.block_scales(stage + G.sc_off);
        ld.ch++;
    }
    cp_async_commit();
}

template <int NMAT, int RL, int T, int STEP, int UNROLL>
__device__ __forceinline__ void run_pass(const Q4Job& jb, Loader<NMAT, RL>& ld, const BatchGeom& G, uint8_t* smem,
                                         int r0, int nvalid, int tb) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, u = lane & 7, lrow = lane >> 3;
    constexpr int ISTEP = RL == 4 ? 8 : 16;
    const int r7 = (warp & 1) * 4 + lrow, sr0 = RL == 4 ? (warp >> 1) * 32 + r7 : warp * 4 + lrow;
    const uint32_t m11 = c_nibble_magic[3], m7 = c_magic_2_7;
    const f32x2 nz = pack2u(c_neg_zero, c_neg_zero);
    const uint32_t* tab = (const uint32_t*)(smem + G.table_off) + sr0 * G.tpitch;
    f32x2 acc[RL][T][2];
#pragma unroll
    for (int i = 0; i < RL; i++)
#pragma unroll
        for (int t = 0; t < T; t++) acc[i][t][0] = acc[i][t][1] = pack2(0.0f, 0.0f);
    const int steps = ld.steps, nch = (steps + CH_STEPS - 1) / CH_STEPS;
    int slot = 0;
    for (int ch = 0; ch < nch; ch++) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
        __syncthreads();                                    // the chunk has landed; everyone is done with the one before
        load_chunk<STEP == STEP_FP4 ? FMT_FP4 : FMT_Q4, NMAT, RL>(ld, G, smem + (slot == 0 ? STAGES - 1 : slot - 1) * G.stage_bytes);
        const uint8_t* stage = smem + slot * G.stage_bytes;
        const uint8_t* w = stage + sr0 * CH_BYTES + 2 * u;
        const float* x = (const float*)(stage + G.x_off) + 4 * u;
        const int live = min(CH_STEPS, steps - ch * CH_STEPS);
        // One Q4 quantisation group per iteration in a layer: the four pass sizes of a layer's groups run side by side on an SM, and their code
        // has to come through the instruction cache.  Two Q4 groups: 16 tokens 1167 -> 1125 us in six layers, 64 tokens 2761 -> 2680,
        // two tokens 365 -> 357; one 32-column step: 1125 and 2787.  An NVFP4 group is shorter, two are better there (136 / 139 us for
        // one token).
        const uint32_t r16 = (uint32_t)r7 << 4;
#pragma unroll UNROLL
        for (int g = 0; g < live / 2; g++) {
            const uint32_t o = ((uint32_t)g << 5) ^ r16;
            if constexpr (STEP == STEP_FP4)
                group_step_fp4<RL, T>(w, o, o ^ 16u, stage + G.sc_off + sr0 * 16 + 4 * g + (u >> 2),
                                      (const float*)(smem + G.table_off), x + g * 64, acc, nz);
            else
                group_step<RL, T, STEP == STEP_Q4_LITERAL>(w, o, o ^ 16u, tab + ch * (CH_COLS / 64) + g, ISTEP * G.tpitch,
                                                           x + g * 64, acc, m11, m7, nz);
        }
        slot = slot + 1 == STAGES ? 0 : slot + 1;
    }
    finish_pass<NMAT, RL, T>(jb, r0, nvalid, tb, (float4*)(smem + G.fold_off + warp * RL * FOLD_BYTES),
                             (float*)(smem + G.table_off), sr0, acc);
}

template <int NMAT, int RL, int STEP, int UNROLL>
__device__ __forceinline__ void run_tokens(const Q4Job& jb, Loader<NMAT, RL>& ld, const BatchGeom& G, uint8_t* smem,
                                           int r0, int nvalid, int tb) {
    if (ld.ntok == 4) run_pass<NMAT, RL, 4, STEP, UNROLL>(jb, ld, G, smem, r0, nvalid, tb);
    else if (ld.ntok == 3) run_pass<NMAT, RL, 3, STEP, UNROLL>(jb, ld, G, smem, r0, nvalid, tb);
    else if (ld.ntok == 2) run_pass<NMAT, RL, 2, STEP, UNROLL>(jb, ld, G, smem, r0, nvalid, tb);
    else run_pass<NMAT, RL, 1, STEP, UNROLL>(jb, ld, G, smem, r0, nvalid, tb);
}

// blockIdx: row tile, job, pass of `pass` of the job's tokens
template <int FMT, int NMAT, int RL, int UNROLL>
__global__ void __launch_bounds__(NT, RL == 4 ? 4 : 6)
batch_kernel(const void* __restrict__ jobs, const int* __restrict__ njobs_dev, int C, int jobs_early, int pass) {
    extern __shared__ __align__(128) uint8_t smem[];
    constexpr int ROWS = 4 * RL * WARPS, ROWS_A = ROWS / NMAT;
    // jobs_early: the job table was written at least two launches back, so everything except the activation rows
    // (the previous kernel's output) may be fetched before the dependency wait
    if (!jobs_early) {
        pdl_wait();
        pdl_launch_dependents();
    }
    const int njobs_live = njobs_dev != nullptr ? __ldcg(njobs_dev) : 0x7fffffff;
    if ((int)blockIdx.y >= njobs_live) return;
    __shared__ __align__(16) Q4Job jb;
    float wg = 0.0f;
    if (FMT == FMT_FP4) {                                   // the same descriptor in the shared form
        const Fp4Job* f = (const Fp4Job*)jobs + blockIdx.y;      // through L2: this SM's L1 may hold an earlier pass' jobs
        wg = __ldcg(&f->wg);
        if (threadIdx.x == 0) {
            static_assert(sizeof(void*) == 8, "pointers as 64-bit words");
            const auto pointer = [](const void* at) { return (void*)__ldcg((const unsigned long long*)at); };
            jb.vals = (const uint8_t*)pointer(&f->codes); jb.scales = (const uint8_t*)pointer(&f->scales);
            jb.x = (const float*)pointer(&f->x); jb.y = (float*)pointer(&f->y); jb.x_rows = nullptr;
            jb.R = __ldcg(&f->R); jb.ntok = __ldcg(&f->ntok); jb.x_stride = __ldcg(&f->x_stride); jb.y_stride = __ldcg(&f->y_stride);
        }
    } else if (threadIdx.x < sizeof(Q4Job) / 16) {
        ((uint4*)&jb)[threadIdx.x] = __ldcg((const uint4*)((const Q4Job*)jobs + blockIdx.y) + threadIdx.x);
    }
    __syncthreads();
    const int r0 = blockIdx.x * ROWS_A, tb = blockIdx.z * pass;
    if (r0 >= jb.R || tb >= jb.ntok) return;
    const int nvalid = min(ROWS_A, jb.R - r0), tid = threadIdx.x;
    const BatchGeom G = batch_geom(FMT, C, NMAT, RL);
    __shared__ const float* x_row[MAX_T];
    Loader<NMAT, RL> ld(jb, x_row, r0, C, min(pass, jb.ntok - tb));

    // first stages: weights and scales, then (after the dependency) activations
    ld.weights(smem);
    if (FMT == FMT_FP4) {
        ld.block_scales(smem + G.sc_off);
        for (int c = tid; c < 256; c += NT) ((float*)(smem + G.table_off))[c] = __fmul_rn(e4m3_decode((uint32_t)c), wg);
    } else {
#pragma unroll
        for (int m = 0; m < NMAT; m++) {
            const uint8_t* gs = (m == 0 ? jb.scales : jb.scales2) + (size_t)r0 * G.raw_pitch;
            const uint8_t* gb = m == 0 ? jb.biases : jb.biases2;
            uint8_t* ds = smem + G.raw_off + 2 * m * G.raw_block;
            uint8_t* db = ds + G.raw_block;
            const int total = nvalid * G.raw_pitch, full = total >> 4;
            if (gb) gb += (size_t)r0 * G.raw_pitch;
            for (int p = tid; p < full; p += NT) {
                cp_async16(ds + p * 16, gs + p * 16);
                if (gb) cp_async16(db + p * 16, gb + p * 16);
            }
            for (int i = (full << 4) + 2 * tid; i < total; i += 2 * NT) {
                *(uint16_t*)(ds + i) = *(const uint16_t*)(gs + i);
                if (gb) *(uint16_t*)(db + i) = *(const uint16_t*)(gb + i);
            }
            if (!gb)
                for (int i = tid; i < G.raw_block / 4; i += NT) ((uint32_t*)db)[i] = 0u;
        }
    }
    if (jobs_early) {
        pdl_wait();
        pdl_launch_dependents();
    }
    if (tid < ld.ntok) {
        const int row = jb.x_rows ? jb.x_rows[tb + tid] / jb.x_div : tb + tid;
        x_row[tid] = jb.x + (size_t)row * jb.x_stride;
    }
    __syncthreads();
    ld.activations(smem + G.x_off);
    ld.ch++;
    cp_async_commit();
#pragma unroll
    for (int k = 1; k < STAGES - 1; k++) load_chunk<FMT, NMAT, RL>(ld, G, smem + k * G.stage_bytes);
    if constexpr (FMT == FMT_FP4) {
        run_tokens<NMAT, RL, STEP_FP4, UNROLL>(jb, ld, G, smem, r0, nvalid, tb);
    } else {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
        __syncthreads();
        // interleave scales and biases; does any group need the two-rounding dequantisation?
        uint32_t key = 0, top = 0;                          // largest near_key and scale of this thread's groups
        uint32_t* table = (uint32_t*)(smem + G.table_off);
        const int gpr = C >> 6;
        for (int sr = tid >> 3; sr < ROWS; sr += NT / 8) {
            const int m = NMAT == 2 ? (sr >> 4) & 1 : 0, lr = tile_row<NMAT>(sr);
            const uint8_t* ds = smem + G.raw_off + 2 * m * G.raw_block + lr * G.raw_pitch;
            for (int g = tid & 7; g < gpr; g += 8) {
                uint32_t hs = 0, hb = 0;
                if (lr < nvalid) {
                    hs = *(const uint16_t*)(ds + 2 * g);
                    hb = *(const uint16_t*)(ds + G.raw_block + 2 * g);
                    key = max(key, near_key(hs, hb));
                    top = max(top, hs & 0x7f80u);
                }
                table[sr * G.tpitch + g] = (hs << 16) | hb;
            }
        }
        int lit = __syncthreads_or(key > NEAR_MAX || top > SCALE_MAX);
        if (lit) {
            lit = 0;
            for (int sr = tid >> 3; sr < ROWS; sr += NT / 8)
                for (int g = tid & 7; g < gpr; g += 8) {
                    const uint32_t word = table[sr * G.tpitch + g];
                    lit |= one_rounding(word >> 16, word & 0xffffu) ? 0 : 1;
                }
            lit = __syncthreads_or(lit);
        }
        if (lit) run_tokens<NMAT, RL, STEP_Q4_LITERAL, UNROLL>(jb, ld, G, smem, r0, nvalid, tb);
        else run_tokens<NMAT, RL, STEP_Q4, UNROLL>(jb, ld, G, smem, r0, nvalid, tb);
    }
}

template <int FMT, int NMAT, int RL, int UNROLL = FMT == FMT_FP4 ? 2 : 1>
cudaError_t launch_batch(const void* jobs, int njobs_max, const int* njobs_dev, int max_rows, int max_tok, int C,
                         cudaStream_t stream, int pdl, int pass = MAX_T) {
    const BatchGeom G = batch_geom(FMT, C, NMAT, RL);
    cudaError_t e = ensure_dynamic_smem((const void*)batch_kernel<FMT, NMAT, RL, UNROLL>, G.smem);
    if (e != cudaSuccess) return e;
    constexpr int ROWS_A = 4 * RL * WARPS / NMAT;
    const dim3 grid((max_rows + ROWS_A - 1) / ROWS_A, njobs_max, (max_tok + pass - 1) / pass);
    if (grid.y > 65535 || grid.z > 65535) return cudaErrorInvalidValue;
    if (pdl >= 0)
        return launch_pdl(batch_kernel<FMT, NMAT, RL, UNROLL>, grid, dim3(NT), (size_t)G.smem, stream, jobs, njobs_dev, C, pdl, pass);
    batch_kernel<FMT, NMAT, RL, UNROLL><<<grid, NT, G.smem, stream>>>(jobs, njobs_dev, C, 0, pass);
    return launched();
}

// Rows per lane.  Four need a quarter of the shared loads per product; two make twice as many blocks, which start and
// end more evenly.  `blocks`: of four rows per lane in the grid (the most that the jobs of the batch can make).  Q4: two are
// better below about thirteen blocks per SM (2 tokens of the layer above 76 -> 72 us; one 4096 x 4096 row product from the host
// 62 -> 51).  NVFP4: below about six: 1536 rows x 5120 x 7 tokens from the host
// 61 -> 49 us, 6144 x 5120 x 32 (5.2 blocks per SM) 254 -> 247; layers (5120 x 1536, top-4) 1 token 88 -> 82 us, 3 tokens (6.5)
// 138 with four against 140, 8 tokens 218 / 226.  One row per lane was slower still.
bool two_rows_per_lane(int fmt, long blocks) { return blocks < (fmt == FMT_Q4 ? 13L : 6L) * device_sms(); }

}  // namespace

bool q4_batch_supported(int C, int nmat) { return C >= 64 && (C % 64) == 0 && batch_geom(FMT_Q4, C, nmat, 4).smem <= 225 * 1024; }

cudaError_t launch_q4_batch(const Q4Job* jobs, int njobs_max, const int* njobs_dev, int max_rows, int max_tok, int C,
                            int nmat, cudaStream_t stream, int pdl, bool alone) {
    const long blocks = (long)((max_rows + 64 / nmat - 1) / (64 / nmat)) * njobs_max * ((max_tok + MAX_T - 1) / MAX_T);
    const bool two = two_rows_per_lane(FMT_Q4, blocks);
#define SB_BATCH(NM, RL) launch_batch<FMT_Q4, NM, RL>(jobs, njobs_max, njobs_dev, max_rows, max_tok, C, stream, pdl)
    // One projection by itself, few blocks: its code does not share the instruction cache with another variant's, two groups per
    // iteration are the shorter loop (from the host, one / two groups: 4096 x 4096 1 token 29.6 / 29.1 us, 4 tokens 61.9 / 60.2, 16 tokens
    // 119 / 118).  Behind a gate/up launch they are not: chain of four one-token experts 40.9 / 42.3, whole block of 4 tokens 149.0 / 150.7.
    if (nmat == 1 && two && alone)
        return launch_batch<FMT_Q4, 1, 2, 2>(jobs, njobs_max, njobs_dev, max_rows, max_tok, C, stream, pdl);
    if (nmat == 2) return two ? SB_BATCH(2, 2) : SB_BATCH(2, 4);
    return two ? SB_BATCH(1, 2) : SB_BATCH(1, 4);
#undef SB_BATCH
}

bool fp4_batch_supported(int C) { return C >= 256 && (C % 256) == 0; }

cudaError_t launch_fp4_batch(const Fp4Job* jobs, int njobs_max, const int* njobs_dev, int max_rows, int max_tok, int C,
                             cudaStream_t stream) {
    const long blocks = (long)((max_rows + 63) / 64) * njobs_max * ((max_tok + MAX_T - 1) / MAX_T);
    if (!two_rows_per_lane(FMT_FP4, blocks)) return launch_batch<FMT_FP4, 1, 4>(jobs, njobs_max, njobs_dev, max_rows, max_tok, C, stream, 1);
    // Jobs of whole groups (their number is the host's): two tokens a pass where even that leaves room for two blocks per SM: a
    // block's products are a chain of chunks, shorter with fewer tokens.  Jobs numbered on the device are passes already.  From the
    // host, four / two tokens a pass: 1536 rows x 5120, 4 tokens 49.3 / 43.8 us, 7 tokens 52.8 / 51.2; 200 x 5120, 16 tokens 60.8 /
    // 55.5; 6000 x 2048, 7 tokens (five blocks per SM) 46.8 / 49.5.
    const bool two = njobs_dev == nullptr && (long)((max_rows + 31) / 32) * njobs_max * ((max_tok + 1) / 2) <= 2L * device_sms();
    return launch_batch<FMT_FP4, 1, 2>(jobs, njobs_max, njobs_dev, max_rows, max_tok, C, stream, 1, two ? 2 : MAX_T);
}

}  // namespace sb
