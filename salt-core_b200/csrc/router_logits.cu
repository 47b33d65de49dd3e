// Router logits, bit-exact: logits[row][e] = the reference's chain acc = fl(acc + fl(W[e][c] * x[row][c])), columns
// ascending from +0 (reference src/kernels.c:98-106).
//
// A logit is a chain of H dependent adds: at 4.4 cycles each 2816 columns take 6.5 us, and rows x experts chains are all the
// parallelism there is unless a chain is added in pieces, which takes several times the additions.  A warp alone on its scheduler issues in order and every shared load
// holds it for about four cycles (measured: 4.5 cycles per column for add + multiply from registers, 8.8 with a 4-byte
// load per column), so a lane owns whole chains and reads 16 bytes at a time:
//   * few chains (router_logits_chain_kernel): a block per chain, products in shared memory, added by the block in pieces
//     (block_sum_ordered), about 4500 cycles for 2816 columns where one warp's chain took 13 000, or, short ones, by one warp.
//   * few rows (router_logits_few_kernel): eight experts x eight rows per block.  Helper warps form the products of a slab
//     of 128 columns and leave them in shared memory, a chain per row; a lane of an adding warp reads four products and
//     does four adds, nothing else.  Few experts per block because a block's weights all come through one SM.
//   * many rows (router_logits_many_kernel): 64 experts x CW R rows per block, NSL x R chains per lane, so that a 16-byte
//     load of weights serves R chains and one of activations NSL.
// Slabs of weights and activations are fetched by warps of their own.  Between events, 128 experts x 2816 columns: 64 rows
// 39 -> 19 us, 512 rows 47 -> 36, 2048 rows 100 -> 76 against tiles of 8 x 8 to 32 x 32 chains, one or four per lane, with a
// barrier per slab.
#include "internal.h"
#include "mbar.cuh"
#include "pdl.cuh"
#include "q4_core.cuh"
#include "router_core.cuh"

namespace sb {
namespace {

constexpr int SLAB = 128;                     // columns (the last slab of a row may be half of that)
constexpr uint32_t SPIN_LIMIT = 1u << 22;
constexpr int PITCH = SLAB + 4;               // floats: rows read side by side start four banks apart
constexpr uint32_t ROW_BYTES = PITCH * 4;

// One look at a barrier's phase.  Used ahead of time: the answer takes some 150 cycles, which other work can cover.
__device__ __forceinline__ bool phase_done(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ bool wait_phase(uint64_t* bar, uint32_t parity) {
    const uint32_t addr = smem_u32(bar);
#pragma unroll 1
    for (uint32_t i = 0; i < SPIN_LIMIT; i++) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(ok)
            : "r"(addr), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// All of this thread's cp.async so far arrive on `bar` once they have landed.
__device__ __forceinline__ void arrive_when_copied(uint64_t* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mul_now(float& p, float a, float b) { asm volatile("mul.rn.f32 %0, %1, %2;" : "=f"(p) : "f"(a), "f"(b)); }

// A fetching warp: slab after slab of `n` rows of src (from row r0, the last one being `last`) into rows `at`, at + 1, ... of
// a ring of `stages` stages of stage_bytes, one row (512 bytes, a 16-byte cp.async per lane) per instruction.  (Bulk
// copies issued from a warp's lanes took about 100 cycles each: the ring ran dry.)  Adds 32 arrivals to full[] per slab.
// `early` slabs do not depend on the previous kernel.  Returns false when a wait ran out.
__device__ __forceinline__ bool fetch_slabs(uint8_t* smem, uint64_t* full, uint64_t* empty, int stages, uint32_t stage_bytes, int at,
                                            int n, const float* __restrict__ src, int r0, int last, int H, int early) {
    const int lane = threadIdx.x & 31, nslab = (H + SLAB - 1) / SLAB;
    const float* p = src + (size_t)min(r0, last) * H + lane * 4;
    const size_t step = r0 + n - 1 <= last ? (size_t)H : 0;  // rows past the end: the last one again
    auto fetch = [&](int sl) {
        uint8_t* dst = smem + (sl % stages) * stage_bytes + at * ROW_BYTES + lane * 16;
        if (sl * SLAB + lane * 4 < H) {
            const float* q = p + sl * SLAB;
            if (step) {
#pragma unroll 8
                for (int i = 0; i < n; i++) cp_async16(dst + i * ROW_BYTES, q + i * step);
            } else {
                for (int i = 0; i < n; i++) cp_async16(dst + i * ROW_BYTES, src + (size_t)min(r0 + i, last) * H + sl * SLAB + lane * 4);
            }
        }
        arrive_when_copied(full + sl % stages);
    };
    early = min(early, min(nslab, stages));
    for (int sl = 0; sl < early; sl++) fetch(sl);
    pdl_wait();
    pdl_launch_dependents();
#pragma unroll 1
    for (int sl = early; sl < nslab; sl++) {
        if (sl >= stages && !wait_phase(empty + sl % stages, (uint32_t)(sl / stages - 1) & 1u)) {
            cp_async_commit();
            cp_async_wait_dyn(0);
            return false;
        }
        fetch(sl);
    }
    return true;
}

// acc += p[0], p[1], ... p[COLS - 1], in order: 32 columns are loaded while the 32 before them are added.  (The bounds are
// compile-time constants: with run-time ones the loads were not kept ahead, 11 cycles per column instead of 4.1.)
// `ahead` runs before the last 32 adds.
template <int COLS, class Ahead>
__device__ __forceinline__ void add_products(const float* p, float& acc, Ahead ahead) {
    float4 v[2][8];
#pragma unroll
    for (int i = 0; i < 8; i++) v[0][i] = load_now(p + 4 * i);
#pragma unroll
    for (int c = 0; c < COLS / 32; c++) {
        if (c + 1 < COLS / 32) {
#pragma unroll
            for (int i = 0; i < 8; i++) v[(c + 1) & 1][i] = load_now(p + 32 * (c + 1) + 4 * i);
        } else {
            ahead();
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
            add_now(acc, v[c & 1][i].x);
            add_now(acc, v[c & 1][i].y);
            add_now(acc, v[c & 1][i].z);
            add_now(acc, v[c & 1][i].w);
        }
    }
}

// ---- few rows: 8 experts x 8 rows per block ------------------------------------------------------------
constexpr int FEW_E = 8, FEW_ROWS = 8, FEW_STAGES = 8;
constexpr uint32_t FEW_STAGE_BYTES = (FEW_E + FEW_ROWS) * ROW_BYTES, FEW_PROD_BYTES = 32 * ROW_BYTES;
constexpr int FEW_BUFS = 4;                   // product buffers of a pair: a helper is a slab ahead when the chains ask for it
constexpr uint32_t FEW_SMEM = FEW_STAGES * FEW_STAGE_BYTES + 2 * FEW_BUFS * FEW_PROD_BYTES + (2 * FEW_STAGES + 4 * FEW_BUFS) * 8;

// Warps 0, 1: chains of rows 0..3, 4..7 (lane = expert + 8 * row); 2, 3: their products of even slabs, 6, 7: of odd slabs
// (a slab takes a helper 640 cycles and about 400 more for its barriers, an adding warp 560); 10, 11: copies.  The other warps
// leave at once: they keep the adding warps alone on their schedulers (beside a helper a slab took 950 cycles).
constexpr int FEW_THREADS = 384;
__global__ void __launch_bounds__(FEW_THREADS, 1)
router_logits_few_kernel(const float* __restrict__ W, const float* __restrict__ x, float* __restrict__ logits, int rows, int E,
                         int H, int* status) {
    extern __shared__ __align__(128) uint8_t smem[];
    uint8_t* prod = smem + FEW_STAGES * FEW_STAGE_BYTES;                        // [2 pairs][FEW_BUFS][32 chains]
    uint64_t* full = (uint64_t*)(prod + 2 * FEW_BUFS * FEW_PROD_BYTES);
    uint64_t *empty = full + FEW_STAGES, *pfull = empty + FEW_STAGES, *pempty = pfull + 2 * FEW_BUFS;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, h = warp & 1;
    const int e0 = blockIdx.x * FEW_E, row0 = blockIdx.y * FEW_ROWS, nslab = (H + SLAB - 1) / SLAB;
    const int pairs = rows - row0 > 4 ? 2 : 1;                                  // adding / helping pairs with rows
    if (threadIdx.x == 0) {
        for (int i = 0; i < FEW_STAGES; i++) {
            mbar_init(full + i, 64);
            mbar_init(empty + i, pairs);
        }
        for (int i = 0; i < 2 * FEW_BUFS; i++) {
            mbar_init(pfull + i, 1);
            mbar_init(pempty + i, 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    bool ok = true;
    if (warp == 10) {
        ok = fetch_slabs(smem, full, empty, FEW_STAGES, FEW_STAGE_BYTES, 0, FEW_E, W, e0, E - 1, H, FEW_STAGES);
    } else if (warp == 11) {
        ok = fetch_slabs(smem, full, empty, FEW_STAGES, FEW_STAGE_BYTES, FEW_E, min(FEW_ROWS, rows - row0), x, row0, rows - 1, H, 0);
    } else if (warp < 4 || (warp & 6) == 6) {
        pdl_wait();
        pdl_launch_dependents();
        if (h < pairs && warp >= 2) {
#pragma unroll 1
            for (int sl = warp >> 2; sl < nslab && ok; sl += 2) {
                const int st = sl % FEW_STAGES, buf = h * FEW_BUFS + sl % FEW_BUFS;
                ok = wait_phase(full + st, (uint32_t)(sl / FEW_STAGES) & 1u);
                if (sl >= FEW_BUFS) ok = ok && wait_phase(pempty + buf, (uint32_t)(sl / FEW_BUFS - 1) & 1u);
                if (4 * lane < H - sl * SLAB) {
                    const float* w = (const float*)(smem + st * FEW_STAGE_BYTES) + 4 * lane;
                    const float* xs = w + (FEW_E + 4 * h) * PITCH;
                    float* p = (float*)(prod + buf * FEW_PROD_BYTES) + 4 * lane;
                    float4 xv[4];
#pragma unroll
                    for (int r = 0; r < 4; r++) xv[r] = load_now(xs + r * PITCH);
                    float4 wv[FEW_E];
#pragma unroll
                    for (int e = 0; e < FEW_E; e++) wv[e] = load_now(w + e * PITCH);
#pragma unroll
                    for (int e = 0; e < FEW_E; e++) {
                        const float4 q = wv[e];
#pragma unroll
                        for (int r = 0; r < 4; r++)
                            *(float4*)(p + (r * 8 + e) * PITCH) = make_float4(__fmul_rn(q.x, xv[r].x), __fmul_rn(q.y, xv[r].y),
                                                                              __fmul_rn(q.z, xv[r].z), __fmul_rn(q.w, xv[r].w));
                    }
                }
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(pfull + buf);
                    mbar_arrive(empty + st);
                }
            }
        } else if (h < pairs) {
            float acc = 0.0f;
            bool ready = false;
#pragma unroll 1
            for (int sl = 0; sl < nslab && ok; sl++) {
                const int buf = h * FEW_BUFS + sl % FEW_BUFS;
                if (!ready) ok = wait_phase(pfull + buf, (uint32_t)(sl / FEW_BUFS) & 1u);
                auto ahead = [&] { ready = phase_done(pfull + h * FEW_BUFS + (sl + 1) % FEW_BUFS, (uint32_t)((sl + 1) / FEW_BUFS) & 1u); };
                const float* p = (const float*)(prod + buf * FEW_PROD_BYTES) + lane * PITCH;
                if (H - sl * SLAB >= SLAB) add_products<SLAB>(p, acc, ahead);
                else add_products<SLAB / 2>(p, acc, ahead);
                __syncwarp();
                if (lane == 0) mbar_arrive(pempty + buf);
            }
            const int e = e0 + (lane & 7), row = row0 + 4 * h + (lane >> 3);
            if (e < E && row < rows) logits[(size_t)row * E + e] = __fadd_rn(acc, 0.0f);   // the reference adds its (absent) bias
        }
    }
    if (!ok) flag(status, SB_ERR_TIMEOUT);
}

// ---- many rows: 32 NSL experts x CW R rows per block ------------------------------------------------------
template <int NSL, int R, int CW>
struct ManyTile {
    static constexpr int WE = 32 * NSL, ROWS = CW * R, THREADS = 32 * (CW + 2);
    static constexpr uint32_t STAGE_BYTES = (WE + ROWS) * ROW_BYTES;
    static constexpr int STAGES = 3;
    static constexpr uint32_t SMEM = STAGES * STAGE_BYTES + 2 * STAGES * 8;
};

// acc[s][r] += w[s][c] * x[r][c], c = 0, 1, ... COLS - 1: four columns loaded while four are added; all products of a
// column, then its adds (independent chains side by side)
template <int COLS, int NSL, int R>
__device__ __forceinline__ void add_columns(const float* w, const float* x, float (&acc)[NSL][R]) {
    float4 wv[2][NSL], xv[2][R];
    auto load = [&](int buf, int c) {
#pragma unroll
        for (int s = 0; s < NSL; s++) wv[buf][s] = load_now(w + s * 32 * PITCH + c);
#pragma unroll
        for (int r = 0; r < R; r++) xv[buf][r] = load_now(x + r * PITCH + c);
    };
    load(0, 0);
#pragma unroll 2
    for (int c = 0; c < COLS; c += 8) {
#pragma unroll
        for (int b = 0; b < 2; b++) {
            if (c + 4 * b + 4 < COLS) load(b ^ 1, c + 4 * b + 4);
#define SB_COLUMN(m)                                                                                     \
    {                                                                                                    \
        float p[NSL][R];                                                                                 \
        _Pragma("unroll") for (int s = 0; s < NSL; s++) _Pragma("unroll") for (int r = 0; r < R; r++)    \
            mul_now(p[s][r], wv[b][s].m, xv[b][r].m);                                                    \
        _Pragma("unroll") for (int s = 0; s < NSL; s++) _Pragma("unroll") for (int r = 0; r < R; r++)    \
            add_now(acc[s][r], p[s][r]);                                                                 \
    }
            SB_COLUMN(x) SB_COLUMN(y) SB_COLUMN(z) SB_COLUMN(w)
#undef SB_COLUMN
        }
    }
}

// CW warps: R rows each, lane = expert; two more: copies
template <int NSL, int R, int CW>
__global__ void __launch_bounds__(32 * (CW + 2), 1)
router_logits_many_kernel(const float* __restrict__ W, const float* __restrict__ x, float* __restrict__ logits, int rows, int E,
                          int H, int* status) {
    using G = ManyTile<NSL, R, CW>;
    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t* full = (uint64_t*)(smem + G::STAGES * G::STAGE_BYTES);
    uint64_t* empty = full + G::STAGES;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int e0 = blockIdx.x * G::WE, row0 = blockIdx.y * G::ROWS, nslab = (H + SLAB - 1) / SLAB;
    if (threadIdx.x == 0) {
        for (int i = 0; i < G::STAGES; i++) {
            mbar_init(full + i, 64);
            mbar_init(empty + i, CW);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    bool ok = true;
    if (warp == CW) {
        ok = fetch_slabs(smem, full, empty, G::STAGES, G::STAGE_BYTES, 0, G::WE, W, e0, E - 1, H, G::STAGES);
    } else if (warp == CW + 1) {
        ok = fetch_slabs(smem, full, empty, G::STAGES, G::STAGE_BYTES, G::WE, min(G::ROWS, rows - row0), x, row0, rows - 1, H, 0);
    } else {
        pdl_wait();
        pdl_launch_dependents();
        float acc[NSL][R];
#pragma unroll
        for (int s = 0; s < NSL; s++)
#pragma unroll
            for (int r = 0; r < R; r++) acc[s][r] = 0.0f;
#pragma unroll 1
        for (int sl = 0; sl < nslab && ok; sl++) {
            const int st = sl % G::STAGES;
            ok = wait_phase(full + st, (uint32_t)(sl / G::STAGES) & 1u);
            const float* w = (const float*)(smem + st * G::STAGE_BYTES) + lane * PITCH;
            const float* xs = (const float*)(smem + st * G::STAGE_BYTES) + (G::WE + warp * R) * PITCH;
            if (H - sl * SLAB >= SLAB) add_columns<SLAB, NSL, R>(w, xs, acc);
            else add_columns<SLAB / 2, NSL, R>(w, xs, acc);
            __syncwarp();
            if (lane == 0) mbar_arrive(empty + st);
        }
#pragma unroll
        for (int s = 0; s < NSL; s++) {
            const int e = e0 + s * 32 + lane;
#pragma unroll
            for (int r = 0; r < R; r++) {
                const int row = row0 + warp * R + r;
                if (e < E && row < rows) logits[(size_t)row * E + e] = __fadd_rn(acc[s][r], 0.0f);
            }
        }
    }
    if (!ok) flag(status, SB_ERR_TIMEOUT);
}

template <int NSL, int R, int CW>
cudaError_t launch_many(const float* W, const float* x, float* logits, int rows, int E, int H, int* status, cudaStream_t stream) {
    using G = ManyTile<NSL, R, CW>;
    cudaError_t e = ensure_dynamic_smem((const void*)router_logits_many_kernel<NSL, R, CW>, G::SMEM);
    if (e != cudaSuccess) return e;
    const dim3 grid((E + G::WE - 1) / G::WE, (rows + G::ROWS - 1) / G::ROWS);
    return launch_pdl(router_logits_many_kernel<NSL, R, CW>, grid, dim3(G::THREADS), (size_t)G::SMEM, stream, W, x, logits, rows, E, H, status);
}

// ---- few chains: a block per (expert, row).  All its threads form the products, coalesced, in shared memory and add
// them together (block_sum_ordered) or, WARP, one of its warps does, another one in each round of blocks (of `sms`).
constexpr int CHAIN_THREADS = 256;
template <int N4, bool WARP>                  // N4: 16-byte pieces per thread
__global__ void __launch_bounds__(CHAIN_THREADS)
router_logits_chain_kernel(const float* __restrict__ W, const float* __restrict__ x, float* __restrict__ logits, int E, int H, int sms) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ __align__(16) uint32_t scratch[ORDERED_SCRATCH];
    const int e = blockIdx.x, r = blockIdx.y, n4 = H >> 2;
    const float4* w4 = (const float4*)(W + (size_t)e * H);
    const float4* x4 = (const float4*)(x + (size_t)r * H);
    float4 w[N4], v[N4];
#pragma unroll
    for (int i = 0; i < N4; i++) {            // the router weights do not depend on the previous kernel
        const int k = threadIdx.x + i * CHAIN_THREADS;
        if (k < n4) w[i] = __ldg(w4 + k);
    }
    pdl_wait();
    pdl_launch_dependents();
#pragma unroll
    for (int i = 0; i < N4; i++) {
        const int k = threadIdx.x + i * CHAIN_THREADS;
        if (k < n4) v[i] = x4[k];
    }
#pragma unroll
    for (int i = 0; i < N4; i++) {
        const int k = threadIdx.x + i * CHAIN_THREADS;
        if (k < n4)
            ((float4*)smem)[k] = make_float4(__fmul_rn(w[i].x, v[i].x), __fmul_rn(w[i].y, v[i].y), __fmul_rn(w[i].z, v[i].z),
                                             __fmul_rn(w[i].w, v[i].w));
    }
    float acc;
    if constexpr (WARP) acc = block_sum_chain((const float*)smem, H, scratch, (int)((blockIdx.y * gridDim.x + blockIdx.x) / sms) & 3);
    else acc = block_sum_ordered((float*)smem, H, 2, scratch);
    if (threadIdx.x == 0) logits[(size_t)r * E + e] = __fadd_rn(acc, 0.0f);
}

}  // namespace

cudaError_t launch_router_logits(const float* W, const float* x, float* logits, int rows, int E, int H, int* status,
                                 cudaStream_t stream) {
    if (rows < 1) return cudaSuccess;
    if ((H % 64) != 0 || ((((uintptr_t)W) | ((uintptr_t)x)) & 15) != 0) return cudaErrorInvalidValue;
    const int sms = device_sms();
    // A block per chain up to five chains per SM, and up to 2.3 + H / 600 of long ones.  The kernel with a chain per lane takes
    // about as long for one chain as for many (logits and top-k of 1024 / 2816 / 5120 columns: 9 / 16 / 25 us).  A block per chain / that
    // kernel (us, chains per SM): 512 columns 4.3: 6.8 / 7.7, 5.2: 8.3 / 7.8; 1024 columns 4.3: 7.9 / 9.0, 5.2: 10.1 / 9.0; 2048 columns
    // 5.2: 12.3 / 13.0, 6.1: 13.2 / 13.1; 2816 columns 6.9: 15.6 / 16.1, 8.6: 17.5 / 16.2; 4096 columns 8.6: 20.4 / 21.2, 10.4:
    // 23.1 / 21.2; 5120 columns 8.6: 22.5 / 25.3, 10.4: 25.3 / 25.4, 12.1: 27.8 / 25.3.
    const long chains = (long)E * rows;
    if (600 * chains <= (long)sms * (H < 1620 ? 3000 : 1380 + H) && H <= 5 * 4 * CHAIN_THREADS) {
        // One warp's chain leaves the schedulers to the other blocks of the SM, pieces need them: chains are the shorter way up to
        // 832 columns, or 700 and 330 more per chain and SM, while all blocks fit at once.  In pieces / as chains (us, chains per
        // SM): 1024 columns 0.9: 7.2 / 7.4, 2.6: 8.2 / 7.2, 4.3: 9.1 / 7.9; 1536 columns 1.7: 8.0 / 8.4, 2.6: 8.6 / 8.5, 4.3: 10.9 / 10.2;
        // 2048 columns 2.6: 9.1 / 9.9, 3.5: 10.0 / 10.0, 4.3: 10.9 / 10.7, 5.2: 12.3 / 14.8; 2816 columns 4.3: 11.7 / 13.0.
        static_assert(3 * 4 * CHAIN_THREADS >= 700 + 5 * 330, "chains by one warp: three pieces per thread");
        const bool warp = chains <= 5L * sms && (H <= 832 || (H - 700) * (long)sms <= 330 * chains);
        const auto kernel = warp ? router_logits_chain_kernel<3, true>
                                 : (H <= 3 * 4 * CHAIN_THREADS ? router_logits_chain_kernel<3, false> : router_logits_chain_kernel<5, false>);
        return launch_pdl(kernel, dim3(E, rows), dim3(CHAIN_THREADS), (size_t)H * 4, stream, W, x, logits, E, H, sms);
    }
    // one chain per lane while one round of blocks holds them all, then as many per lane as keep it to one round
    const long few = (long)((E + FEW_E - 1) / FEW_E) * ((rows + FEW_ROWS - 1) / FEW_ROWS);
    if (few <= sms) {
        cudaError_t e = ensure_dynamic_smem((const void*)router_logits_few_kernel, FEW_SMEM);
        if (e != cudaSuccess) return e;
        return launch_pdl(router_logits_few_kernel, dim3((E + FEW_E - 1) / FEW_E, (rows + FEW_ROWS - 1) / FEW_ROWS), dim3(FEW_THREADS),
                          (size_t)FEW_SMEM, stream, W, x, logits, rows, E, H, status);
    }
    const long lanes = (long)((E + 31) / 32) * ((rows + 3) / 4);                 // blocks of one chain per lane
    if (lanes <= sms) return launch_many<1, 1, 4>(W, x, logits, rows, E, H, status, stream);
    if (lanes <= 2 * sms) return launch_many<1, 2, 4>(W, x, logits, rows, E, H, status, stream);
    if (lanes <= 4 * sms) return launch_many<2, 2, 4>(W, x, logits, rows, E, H, status, stream);
    // Two adding warps per scheduler: one alone issues an addition or a product every 1.5 to 1.8 cycles, two together one every 1.1
    // to 1.3.  Seven warps where their smaller tiles take no more time in all: 1999 rows 88.5 -> 77.1 us (eight warps 81.8), 1024 rows 49.4
    // -> 45.7 (50.4); 512 rows 34.6 with four warps of four chains per lane, 35.2 with seven of two.
    const auto rounds = [&](int tile) { return ((long)((E + 63) / 64) * ((rows + tile - 1) / tile) + sms - 1) / sms; };
    if (lanes <= 8 * sms) {
        if (7 * rounds(14) <= 8 * rounds(16)) return launch_many<2, 2, 7>(W, x, logits, rows, E, H, status, stream);
        return launch_many<2, 2, 8>(W, x, logits, rows, E, H, status, stream);
    }
    if (7 * rounds(28) <= 8 * rounds(32)) return launch_many<2, 4, 7>(W, x, logits, rows, E, H, status, stream);
    return launch_many<2, 4, 8>(W, x, logits, rows, E, H, status, stream);
}

}  // namespace sb
