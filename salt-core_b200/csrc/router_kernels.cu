// Router, grouping and reduction kernels of the MoE feed-forward path.
//
// Everything here is bit-exact against the reference CPU functions; the reference arithmetic
// contains several chains that are serial by definition (sums of squares, router logits,
// softmax denominators).  Many chains run side by side, each added by a lane; where few are asked for, the whole block
// adds one (block_sum_ordered) or, a short one, one of its warps does.
#include <cooperative_groups.h>
#include "internal.h"
#include "pdl.cuh"
#include "q4_core.cuh"
#include "router_core.cuh"

namespace sb {

// One copy of the in-order sum per kernel: its instructions are fetched cold, and the second sum finds them there.  SHORT: rows
// that one warp adds, kernels of their own: with both ways in one function the launches of a one-token block took 0.5 us longer.
template <bool SHORT>
static __device__ __noinline__ float row_sum_of_squares(float* p, int n, uint32_t* scratch) {
    if constexpr (SHORT) return block_sum_chain(p, n, scratch, 0);
    else return block_sum_ordered(p, n, 1, scratch);
}

// mode 0: RMSNorm  y = (x*inv) [* weight]             (gemma4.c:85-101)
// mode 1: router input  y = ((x*inv)*scale)*root      (gemma4.c:103-130)
template <int MODE, bool SHORT>
__global__ void __launch_bounds__(256)
norm_rows_kernel(const float* __restrict__ x, const float* __restrict__ weight, float* __restrict__ y, int n,
                 float eps, int with_scale, float root_in, int* status) {
    extern __shared__ __align__(16) float srow[];   // [n] row, then [n (padded to 4)] squares
    float* ssq = srow + ((n + 3) & ~3);
    __shared__ float s_inv, s_root;
    __shared__ __align__(16) uint32_t s_scan[ORDERED_SCRATCH];
    const float* xr = x + (size_t)blockIdx.x * n;
    float* yr = y + (size_t)blockIdx.x * n;
    bool bad = false;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const float v = xr[i];
        srow[i] = v;
        ssq[i] = __fmul_rn(v, v);
        bad |= !finite_f(v);
        if (MODE == 1 || with_scale) bad |= !finite_f(weight[i]);
    }
    const float ss = row_sum_of_squares<SHORT>(ssq, n, s_scan);
    if (threadIdx.x == 0) {
        {
            const float mean = __fadd_rn(__fdiv_rn(ss, (float)n), eps);
            const float inv = pow_neg_half(mean);
            float root = 1.0f;
            if (MODE == 1) root = root_in > 0.0f ? root_in : __fdiv_rn(1.0f, sqrtf_exact((float)n));
            s_inv = inv;
            s_root = root;
            if (!finite_f(inv) || !finite_f(root)) flag(status, SB_ERR_NONFINITE);
        }
    }
    __syncthreads();
    const float inv = s_inv, root = s_root;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        float v = __fmul_rn(srow[i], inv);
        if (MODE == 1) {
            v = __fmul_rn(v, weight[i]);
            v = __fmul_rn(v, root);
        } else if (with_scale) {
            v = __fmul_rn(v, weight[i]);
        }
        bad |= !finite_f(v);
        yr[i] = v;
    }
    if (bad) flag(status, SB_ERR_NONFINITE);
}

// Token-wise glue between the expert phase of one layer and the router of the
// next, in one launch per row:
//   [reduce]  v = ordered weighted sum of the row's grouped expert outputs
//             (src/tensorops.c:291-325), else v = x_in
//   [norm]    v = RMSNorm(v) * norm_w                      (gemma4.c:85-101)
//             y_out = v  (written whenever reduce or norm ran)
//   [router]  rin = ((v * inv) * scale) * (1/sqrt(n))      (gemma4.c:103-130)
// The two sums of squares are formed in element order over squares computed in
// parallel (row_sum_of_squares).
// ---- affine 8-bit matvec (router projections of packages that quantise the router) -----------
// src/kernels.c:343-369: one byte per element, bf16 scale / bias per 64 consecutive elements of
// the flattened matrix (rows may straddle groups), ONE serial chain per row:
// acc = fl(acc + fl(d * x[c])), d = fl(fl(q*s) + b).  One block per (row, token, job): the
// products are formed in parallel, one thread runs the chain.
__global__ void __launch_bounds__(128) q8_rows_kernel(const Q4Job* __restrict__ jobs) {
    extern __shared__ __align__(16) float q8_sm[];
    const Q4Job jb = jobs[blockIdx.z];
    const int r = blockIdx.x, tok = blockIdx.y;
    if (r >= jb.R || tok >= jb.ntok) return;
    const float* x = jb.x + (size_t)tok * jb.x_stride;
    const size_t k0 = (size_t)r * (size_t)jb.C;
    for (int c = threadIdx.x; c < jb.C; c += blockDim.x) {
        const size_t k = k0 + (size_t)c, g = k >> 6;
        const float s = bf16_bits_to_f32(((const uint16_t*)jb.scales)[g]);
        const float b = jb.biases ? bf16_bits_to_f32(((const uint16_t*)jb.biases)[g]) : 0.0f;
        const float d = __fadd_rn(__fmul_rn((float)jb.vals[k], s), b);
        q8_sm[c] = __fmul_rn(d, x[c]);
    }
    __syncthreads();
    if (threadIdx.x == 0) jb.y[(size_t)tok * jb.y_stride + r] = serial_sum(q8_sm, jb.C);
}

cudaError_t launch_q8_jobs(const Q4Job* jobs, int njobs, int max_rows, int max_tok, int C, cudaStream_t stream) {
    if (njobs < 1 || max_rows < 1 || max_tok < 1) return cudaSuccess;
    const size_t smem = (size_t)((C + 3) & ~3) * sizeof(float);
    if (smem > 200 * 1024 || max_tok > 65535 || njobs > 65535) return cudaErrorInvalidValue;
    if (smem > 48 * 1024) {
        cudaError_t e = ensure_dynamic_smem((const void*)q8_rows_kernel, (size_t)(200 * 1024));
        if (e != cudaSuccess) return e;
    }
    q8_rows_kernel<<<dim3(max_rows, max_tok, njobs), 128, smem, stream>>>(jobs);
    return launched();
}

// ---- consumers of the routed-expert output (exact cells) -------------------------------------
// y = (x * inv) * w with inv = (mean(x^2) + eps)^-1/2, one row per block; sq = n floats of shared
// memory.  Returns with y complete and visible to the whole block.
template <bool SHORT>
static __device__ void norm_row_block(const float* x, const float* w, float* y, int n, float eps, float* sq,
                                      uint32_t* scan, float* s_inv, bool& bad, int* status) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const float v = x[i];
        sq[i] = __fmul_rn(v, v);
        bad |= !finite_f(v) || !finite_f(w[i]);
    }
    const float ss = row_sum_of_squares<SHORT>(sq, n, scan);
    if (threadIdx.x == 0) {
        *s_inv = pow_neg_half(__fadd_rn(__fdiv_rn(ss, (float)n), eps));
        if (!finite_f(*s_inv)) flag(status, SB_ERR_NONFINITE);
    }
    __syncthreads();
    const float inv = *s_inv;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const float t = __fmul_rn(__fmul_rn(x[i], inv), w[i]);
        bad |= !finite_f(t);
        y[i] = t;
    }
    __syncthreads();
}

// out = residual + RMSNorm(branch) * weight   (models/gemma4-26b-a4b/src/gemma4.c:188-213)
template <bool SHORT>
__global__ void __launch_bounds__(1024)
residual_postnorm_rows_kernel(const float* __restrict__ residual, const float* __restrict__ branch,
                              const float* __restrict__ weight, float* __restrict__ out, int n, float eps,
                              int* status) {
    extern __shared__ __align__(16) float cell_sm[];     // [n] squares, [n] normalised branch
    __shared__ float s_inv;
    __shared__ __align__(16) uint32_t s_scan[ORDERED_SCRATCH];
    const size_t row = blockIdx.x;
    float* normed = cell_sm + ((n + 3) & ~3);
    bool bad = false;
    norm_row_block<SHORT>(branch + row * n, weight, normed, n, eps, cell_sm, s_scan, &s_inv, bad, status);
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const float r = residual[row * n + i];
        const float y = __fadd_rn(r, normed[i]);
        bad |= !finite_f(r) || !finite_f(y);
        out[row * n + i] = y;
    }
    if (bad) flag(status, SB_ERR_NONFINITE);
}

// sum = RMSNorm(dense)*wd + RMSNorm(routed)*wr; fin = RMSNorm(sum)*wf; out = (residual + fin) * scalar
// (gemma4.c:215-276).  scratch_a / scratch_b receive sum / fin as the reference leaves them.
template <bool SHORT>
__global__ void __launch_bounds__(1024)
parallel_combine_rows_kernel(const float* __restrict__ residual, const float* __restrict__ dense,
                             const float* __restrict__ routed, const float* __restrict__ wd,
                             const float* __restrict__ wr, const float* __restrict__ wf, float* scratch_a,
                             float* scratch_b, float* __restrict__ out, int n, float eps, float scalar, int* status) {
    extern __shared__ __align__(16) float cell_sm[];     // [n] squares
    __shared__ float s_inv;
    __shared__ __align__(16) uint32_t s_scan[ORDERED_SCRATCH];
    const size_t row = blockIdx.x;
    float* sum = scratch_a + row * n;
    float* fin = scratch_b + row * n;
    bool bad = !finite_f(scalar);
    norm_row_block<SHORT>(dense + row * n, wd, sum, n, eps, cell_sm, s_scan, &s_inv, bad, status);
    norm_row_block<SHORT>(routed + row * n, wr, fin, n, eps, cell_sm, s_scan, &s_inv, bad, status);
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const float c = __fadd_rn(sum[i], fin[i]);
        bad |= !finite_f(c);
        sum[i] = c;
    }
    __syncthreads();
    norm_row_block<SHORT>(sum, wf, fin, n, eps, cell_sm, s_scan, &s_inv, bad, status);
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const float r = residual[row * n + i];
        const float y = __fmul_rn(__fadd_rn(r, fin[i]), scalar);
        bad |= !finite_f(r) || !finite_f(y);
        out[row * n + i] = y;
    }
    if (bad) flag(status, SB_ERR_NONFINITE);
}

// logits = cap * tanh(logits / cap), in place   (gemma4.c:278-286)
__global__ void __launch_bounds__(256) softcap_kernel(float* __restrict__ logits, int n, float cap, int* status) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float v = logits[i];
    if (!finite_f(v)) {
        flag(status, SB_ERR_NONFINITE);
        return;
    }
    logits[i] = __fmul_rn(cap, tanhf_exact(__fdiv_rn(v, cap)));
}

// Shared memory of the kernels that hold whole rows of any width, up to 200 KB of them.
static cudaError_t allow_row_smem(const void* kernel, size_t smem) {
    constexpr size_t most = 200 * 1024;
    if (smem > most) return cudaErrorInvalidValue;
    return smem > PLAIN_DYNAMIC_SMEM ? ensure_dynamic_smem(kernel, most) : cudaSuccess;
}

cudaError_t launch_residual_postnorm(const float* residual, const float* branch, const float* weight, float* out,
                                     int rows, int n, float eps, int* status, cudaStream_t stream) {
    if (rows < 1) return cudaSuccess;
    const size_t smem = (2 * (((size_t)n + 3) & ~(size_t)3) + 8) * sizeof(float);
    const auto kernel = sum_in_chain(n, 1) ? residual_postnorm_rows_kernel<true> : residual_postnorm_rows_kernel<false>;
    const cudaError_t e = allow_row_smem((const void*)kernel, smem);
    if (e != cudaSuccess) return e;
    kernel<<<rows, 1024, smem, stream>>>(residual, branch, weight, out, n, eps, status);
    return launched();
}

cudaError_t launch_parallel_combine(const float* residual, const float* dense, const float* routed, const float* wd,
                                    const float* wr, const float* wf, float* scratch_a, float* scratch_b, float* out,
                                    int rows, int n, float eps, float scalar, int* status, cudaStream_t stream) {
    if (rows < 1) return cudaSuccess;
    const size_t smem = ((size_t)n + 8) * sizeof(float);
    const auto kernel = sum_in_chain(n, 1) ? parallel_combine_rows_kernel<true> : parallel_combine_rows_kernel<false>;
    const cudaError_t e = allow_row_smem((const void*)kernel, smem);
    if (e != cudaSuccess) return e;
    kernel<<<rows, 1024, smem, stream>>>(residual, dense, routed, wd, wr, wf, scratch_a, scratch_b, out, n, eps, scalar, status);
    return launched();
}

cudaError_t launch_softcap(float* logits, int n, float cap, int* status, cudaStream_t stream) {
    if (n < 1) return cudaSuccess;
    softcap_kernel<<<(n + 255) / 256, 256, 0, stream>>>(logits, n, cap, status);
    return launched();
}

// Each thread owns the columns d = threadIdx.x + j * blockDim.x (j < GLUE_NV, compile
// time) so that every global load of a phase is issued before the first use: the norm
// weights and router scales right at the start, the rows of the expert outputs as soon as
// the rank table is known.
// <4, 8> with 1024 threads serves rows up to 4096 columns; <16, 2> with 512 threads up to 8192.
template <int GLUE_NV, int GLUE_RB, bool SHORT>
__global__ void __launch_bounds__(GLUE_NV == 4 ? 1024 : 512) glue_rows_kernel(GlueArgs a) {
    extern __shared__ __align__(16) float gsm[];
    const int n = a.n;
    float* sq = gsm;                       // [n] squares for the ordered sums
    __shared__ float s_inv, s_root;
    __shared__ __align__(16) uint32_t s_scan[ORDERED_SCRATCH];
    __shared__ int s_g[64];
    __shared__ float s_w[64];
    const int row = blockIdx.x, T = blockDim.x, tid = threadIdx.x;
    bool bad = false;
    float v[GLUE_NV], nw[GLUE_NV], rs[GLUE_NV];
#pragma unroll
    for (int j = 0; j < GLUE_NV; j++) {
        const int d = tid + j * T;
        nw[j] = (a.norm_w != nullptr && d < n) ? __ldg(a.norm_w + d) : 1.0f;
        rs[j] = (a.router_scale != nullptr && d < n) ? __ldg(a.router_scale + d) : 1.0f;
        v[j] = 0.0f;
    }
    if (tid == 32) s_root = __fdiv_rn(1.0f, sqrtf_exact((float)n));     // beside the loads, not in the chain below
    // the rank table was written by the plan kernel, at least two launches back (unless tables_late)
    int early_g = -1;
    float early_w = 0.0f;
    if (a.grouped != nullptr && tid < a.topk && !a.tables_late) {
        early_g = __ldcg(a.c2g + row * a.topk + tid);      // through L2: this SM's L1 may hold an earlier pass
        early_w = __ldcg(a.weights + row * a.topk + tid);
    }
    pdl_wait();                    // the expert outputs (or x_in) come from the previous kernel
    pdl_launch_dependents();
    if (a.grouped != nullptr && tid < a.topk && a.tables_late) {
        early_g = __ldcg(a.c2g + row * a.topk + tid);
        early_w = __ldcg(a.weights + row * a.topk + tid);
    }
    if (a.grouped != nullptr) {
        // rank -> (grouped row, weight) once per block; invalid ranks are dropped and flagged
        if (tid < a.topk) {
            int g = early_g;
            const float w = early_w;
            if (g < 0 || g >= a.jobs || !finite_f(w)) {
                flag(a.status, g < 0 || g >= a.jobs ? SB_ERR_INDEX : SB_ERR_NONFINITE);
                g = -1;
            }
            s_g[tid] = g;
            s_w[tid] = w;
        }
        __syncthreads();
        for (int r0 = 0; r0 < a.topk; r0 += GLUE_RB) {
            float o[GLUE_NV][GLUE_RB];
#pragma unroll
            for (int i = 0; i < GLUE_RB; i++) {
                const int g = r0 + i < a.topk ? s_g[r0 + i] : -1;
#pragma unroll
                for (int j = 0; j < GLUE_NV; j++) {
                    const int d = tid + j * T;
                    o[j][i] = (g >= 0 && d < n) ? __ldg(a.grouped + (size_t)g * n + d) : 0.0f;
                }
            }
#pragma unroll
            for (int i = 0; i < GLUE_RB; i++)
                if (r0 + i < a.topk && s_g[r0 + i] >= 0) {
                    const float w = s_w[r0 + i];
#pragma unroll
                    for (int j = 0; j < GLUE_NV; j++) v[j] = __fadd_rn(v[j], __fmul_rn(w, o[j][i]));
                }
        }
    } else {
#pragma unroll
        for (int j = 0; j < GLUE_NV; j++) {
            const int d = tid + j * T;
            if (d < n) v[j] = a.x_in[(size_t)row * n + d];
        }
    }
    if (a.norm_w != nullptr) {
#pragma unroll
        for (int j = 0; j < GLUE_NV; j++) {
            const int d = tid + j * T;
            if (d < n) {
                sq[d] = __fmul_rn(v[j], v[j]);
                bad |= !finite_f(v[j]) || !finite_f(nw[j]);
            }
        }
        const float ss = row_sum_of_squares<SHORT>(sq, n, s_scan);
        if (tid == 0) {
            s_inv = pow_neg_half(__fadd_rn(__fdiv_rn(ss, (float)n), a.eps_norm));
            if (!finite_f(s_inv)) flag(a.status, SB_ERR_NONFINITE);
        }
        __syncthreads();
        const float inv = s_inv;
#pragma unroll
        for (int j = 0; j < GLUE_NV; j++) {
            v[j] = __fmul_rn(__fmul_rn(v[j], inv), nw[j]);
            if (tid + j * T < n) bad |= !finite_f(v[j]);
        }
    }
    if (a.y_out != nullptr) {
#pragma unroll
        for (int j = 0; j < GLUE_NV; j++) {
            const int d = tid + j * T;
            if (d < n) a.y_out[(size_t)row * n + d] = v[j];
        }
    }
    if (a.router_scale != nullptr) {
        __syncthreads();   // the previous ordered sum has been read by everyone before sq is rewritten
#pragma unroll
        for (int j = 0; j < GLUE_NV; j++) {
            const int d = tid + j * T;
            if (d < n) {
                sq[d] = __fmul_rn(v[j], v[j]);
                bad |= !finite_f(v[j]) || !finite_f(rs[j]);
            }
        }
        const float ss = row_sum_of_squares<SHORT>(sq, n, s_scan);
        if (tid == 0) {
            s_inv = pow_neg_half(__fadd_rn(__fdiv_rn(ss, (float)n), a.eps_router));
            if (!finite_f(s_inv) || !finite_f(s_root)) flag(a.status, SB_ERR_NONFINITE);
        }
        __syncthreads();
        const float inv = s_inv, root = s_root;
#pragma unroll
        for (int j = 0; j < GLUE_NV; j++) {
            const int d = tid + j * T;
            if (d < n) {
                const float t = __fmul_rn(__fmul_rn(__fmul_rn(v[j], inv), rs[j]), root);
                bad |= !finite_f(t);
                a.rin[(size_t)row * n + d] = t;
            }
        }
    }
    if (bad) flag(a.status, SB_ERR_NONFINITE);
}

// The same glue for batches of several hundred rows: a warp per row, four rows per block.  Lane l holds 16-byte pieces l,
// l + 32, ... of its row in registers.  The squares of the four rows go to shared memory and ONE warp runs the four
// in-order sums side by side, a row per lane (the reference's order: columns ascending from +0).  A chain of 2816 costs about
// 6 us, but the rows of a few blocks per SM run side by side, where the block-per-row form above keeps a whole SM busy for
// 10 us per row with two sums.  (Rows in lane-contiguous pieces, the sum handed from lane to lane, loaded 32 lines per
// instruction: 1999 rows took 68 us for reduce and two sums, this takes 56.)
// P: pieces per lane, an even number, for rows of more than 128 (P - 2) and at most 128 P columns; FULL: exactly 128 P.  The
// row takes 4 P registers of a lane and what is left of its share holds the loads in flight, and pieces that may lie outside
// the row cost a test each: with P in steps of eight, 320 to 592 rows of 2816 columns took 35 us against 30, 256 rows of 5120
// 43 us, with tests of the last two pieces 41, without 39.  Blocks per SM (of registers): four up to 22 pieces, two above 24,
// where three left so few loads in flight that 512 rows of 4096 columns took 46 us against 36.
constexpr int GLUE_ROWS = 4;
constexpr int GLUE_PIECES = 48;            // most: 192 registers, two blocks per SM
static __device__ __forceinline__ uint32_t glue_pitch(int n) { return (uint32_t)n + 4u; }    // the rows start four banks apart

// Does the lane's piece i lie inside the row?  FULL: the row has exactly 128 P columns.
template <int P, bool FULL>
static __device__ __forceinline__ bool glue_in_row(int i, int lane, int n) { return FULL || i < P - 2 || 4 * (lane + 32 * i) < n; }

// Squares of the warps' rows in sq[GLUE_ROWS][pitch] -> s_inv[r] = pow(sum / n + eps, -0.5) for every row of the block.
template <int P, bool FULL>
static __device__ __forceinline__ void glue_inv_rms(const float4 (&v)[P], float* sq, float* s_inv, int n, float eps, int sms) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float4* mine = (float4*)(sq + w * glue_pitch(n)) + lane;
#pragma unroll
    for (int i = 0; i < P; i++)
        if (glue_in_row<P, FULL>(i, lane, n))
            mine[32 * i] = make_float4(__fmul_rn(v[i].x, v[i].x), __fmul_rn(v[i].y, v[i].y), __fmul_rn(v[i].z, v[i].z), __fmul_rn(v[i].w, v[i].w));
    __syncthreads();
    if (w == ((blockIdx.x / sms) & 3)) {          // blocks that share an SM add on different schedulers
        const float ss = chain_sum(sq + (lane & 3) * glue_pitch(n), n);
        if (lane < GLUE_ROWS) s_inv[lane] = pow_neg_half(__fadd_rn(__fdiv_rn(ss, (float)n), eps));
    }
    __syncthreads();
}

static __device__ __forceinline__ bool all_finite(const float4& v) { return finite_f(v.x) && finite_f(v.y) && finite_f(v.z) && finite_f(v.w); }

template <int P, bool FULL>
__global__ void __launch_bounds__(32 * GLUE_ROWS, P <= 22 ? 4 : (P <= 24 ? 3 : 2)) glue_rows_warp_kernel(GlueArgs a, int rows, int sms) {
    static_assert(GLUE_ROWS == 4, "four schedulers");
    extern __shared__ __align__(16) float gsm[];
    __shared__ float s_inv[GLUE_ROWS];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const bool live = blockIdx.x * GLUE_ROWS + w < rows;            // rows past the end: the last one again, not stored
    const int row = live ? blockIdx.x * GLUE_ROWS + w : rows - 1;
    const int n = FULL ? 128 * P : a.n;
    bool bad = false;
    float4 v[P];
#pragma unroll
    for (int i = 0; i < P; i++) v[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (a.grouped != nullptr) {
        for (int r = 0; r < a.topk; r++) {
            const int g = a.c2g[row * a.topk + r];
            const float f = a.weights[row * a.topk + r];
            if (g < 0 || g >= a.jobs || !finite_f(f)) {
                if (lane == 0) flag(a.status, g < 0 || g >= a.jobs ? SB_ERR_INDEX : SB_ERR_NONFINITE);
                continue;
            }
            const float4* src = (const float4*)(a.grouped + (size_t)g * n) + lane;
#pragma unroll
            for (int i = 0; i < P; i++)
                if (glue_in_row<P, FULL>(i, lane, n)) {
                    const float4 o = __ldg(src + 32 * i);
                    v[i].x = __fadd_rn(v[i].x, __fmul_rn(f, o.x));
                    v[i].y = __fadd_rn(v[i].y, __fmul_rn(f, o.y));
                    v[i].z = __fadd_rn(v[i].z, __fmul_rn(f, o.z));
                    v[i].w = __fadd_rn(v[i].w, __fmul_rn(f, o.w));
                }
        }
    } else {
        const float4* src = (const float4*)(a.x_in + (size_t)row * n) + lane;
#pragma unroll
        for (int i = 0; i < P; i++)
            if (glue_in_row<P, FULL>(i, lane, n)) v[i] = src[32 * i];
    }
    if (a.norm_w != nullptr) {
        glue_inv_rms<P, FULL>(v, gsm, s_inv, n, a.eps_norm, sms);
        const float inv = s_inv[w];
        if (!finite_f(inv) && lane == 0) flag(a.status, SB_ERR_NONFINITE);
        const float4* nw4 = (const float4*)a.norm_w + lane;
#pragma unroll
        for (int i = 0; i < P; i++)
            if (glue_in_row<P, FULL>(i, lane, n)) {
                const float4 m = __ldg(nw4 + 32 * i);
                bad |= !all_finite(v[i]) || !all_finite(m);
                v[i].x = __fmul_rn(__fmul_rn(v[i].x, inv), m.x);
                v[i].y = __fmul_rn(__fmul_rn(v[i].y, inv), m.y);
                v[i].z = __fmul_rn(__fmul_rn(v[i].z, inv), m.z);
                v[i].w = __fmul_rn(__fmul_rn(v[i].w, inv), m.w);
            }
    }
    if (a.y_out != nullptr && live) {
        float4* dst = (float4*)(a.y_out + (size_t)row * n) + lane;
#pragma unroll
        for (int i = 0; i < P; i++)
            if (glue_in_row<P, FULL>(i, lane, n)) dst[32 * i] = v[i];
    }
    if (a.router_scale != nullptr) {
        glue_inv_rms<P, FULL>(v, gsm, s_inv, n, a.eps_router, sms);
        const float inv = s_inv[w], root = __fdiv_rn(1.0f, sqrtf_exact((float)n));
        if ((!finite_f(inv) || !finite_f(root)) && lane == 0) flag(a.status, SB_ERR_NONFINITE);
        const float4* rs4 = (const float4*)a.router_scale + lane;
        float4* dst = (float4*)(a.rin + (size_t)row * n) + lane;
#pragma unroll
        for (int i = 0; i < P; i++)
            if (glue_in_row<P, FULL>(i, lane, n)) {
                const float4 m = __ldg(rs4 + 32 * i);
                float4 t;
                t.x = __fmul_rn(__fmul_rn(__fmul_rn(v[i].x, inv), m.x), root);
                t.y = __fmul_rn(__fmul_rn(__fmul_rn(v[i].y, inv), m.y), root);
                t.z = __fmul_rn(__fmul_rn(__fmul_rn(v[i].z, inv), m.z), root);
                t.w = __fmul_rn(__fmul_rn(__fmul_rn(v[i].w, inv), m.w), root);
                bad |= !all_finite(v[i]) || !all_finite(m) || !all_finite(t);
                if (live) dst[32 * i] = t;
            }
    }
    if (bad) flag(a.status, SB_ERR_NONFINITE);
}

template <int P>
static cudaError_t launch_glue_warps(const GlueArgs& a, int rows, int sms, cudaStream_t stream) {
    if constexpr (P < GLUE_PIECES)
        if (a.n > 128 * P) return launch_glue_warps<P + 2>(a, rows, sms, stream);
    const size_t smem = (size_t)GLUE_ROWS * (a.n + 4) * sizeof(float);
    const auto kernel = a.n == 128 * P ? glue_rows_warp_kernel<P, true> : glue_rows_warp_kernel<P, false>;
    cudaError_t e = ensure_dynamic_smem((const void*)kernel, smem);
    if (e != cudaSuccess) return e;
    kernel<<<(rows + GLUE_ROWS - 1) / GLUE_ROWS, 32 * GLUE_ROWS, smem, stream>>>(a, rows, sms);
    return launched();
}

// Most rows for which the block-per-row form is the faster one.  It takes a full round of the chip for every round of blocks (one
// per SM; four of 256 threads for rows up to 1024 columns), the warp form about as long for one row as for several hundred.
// Measured with 148 SMs, four / eight selections (one launch, us, block against warp form):
//   two sums: 64 columns 592 rows 6.3 against 6.7 / 6.5 against 6.7, 740 rows 8.8 against 6.8; 1024 columns 592 rows 12.4 against
//   11.6 / 12.7 against 12.6; 1536 columns 160 rows 16.8 against 14.7 / 18.3 against 16.7; 1792 columns 160 rows - / 17.4 against 18.8;
//   2816 columns 296 rows 19.2 against 26.3 / 20.2 against 29.0, 320 rows 27.3 against 26.8 / 28.4 against 29.3; 4096 columns 444
//   rows 30.8 against 31.1 / 33.1 against 35.1; 4160 columns 296 rows 25.4 against 31.1, 320 rows 34.4 against 31.0; 5120 columns 296
//   rows 25.8 against 37.2 / 31.5 against 39.3, 320 rows 35.9 against 37.1 / 43.2 against 39.3; 6144 columns 444 rows 40.7 against 47.1 /
//   54.8 against 66.0, 480 rows 50.9 against 47.5 / 69.1 against 70.0;
//   one sum: 1024 columns 592 rows 8.7 against 8.5 / 8.4 against 10.3; 2048 columns 160 rows 12.1 against 12.6 / 12.9 against 14.6,
//   256 rows 13.3 against 12.6 / 13.9 against 14.6; 2816 columns 296 rows 13.8 against 16.7 / 14.8 against 20.8, 320 rows 19.2 against
//   16.8 / 19.6 against 20.8; 5120 columns 296 rows 17.7 against 22.9 / 22.3 against 24.9; 6144 columns 444 rows 27.0 against 29.0 /
//   39.4 against 43.3;
//   no sum: 1024 columns 592 rows 4.4 against 4.5 / 4.9 against 6.5, 888 rows 5.9 against 6.2 / 6.5 against 6.6, 1184 rows 7.2 against
//   6.4 / 8.1 against 6.7; 1088 columns 160 rows 6.6 against 6.3 / 7.1 against 6.4; 2048 columns 296 rows 7.0 against 6.4 / 7.7 against
//   8.5; 2816 columns 296 rows 7.1 against 8.4 / 8.0 against 12.5, 444 rows 10.2 against 8.5 / 11.6 against 12.5; 5120 columns 160
//   rows 8.2 against 8.4 / 12.6 against 10.6; 6144 columns 296 rows 9.0 against 10.6 / 14.4 against 16.7.
static int glue_block_rows(const GlueArgs& a, int sms) {
    const int sums = (a.norm_w != nullptr) + (a.router_scale != nullptr);
    if (sums == 0) {
        const bool many = a.topk > 4;
        if (a.n <= 1024) return (many ? 6 : 4) * sms;
        if (many && a.n > 2048 && a.n <= 2816) return 3 * sms;      // above 2816 columns fewer warp-form blocks share an SM
        return (a.n < 2048 || (a.n == 2048 && !many) || (a.n > 4096 && a.n <= 5120) ? 1 : 2) * sms;
    }
    if (a.n <= 1024) return 4 * sms;
    const int rounds = a.n <= (sums == 2 ? 1664 : 2048) ? 1 : (a.n <= 5120 ? 2 : 3);
    return rounds * sms;
}

cudaError_t launch_glue(const GlueArgs& a, int rows, cudaStream_t stream) {
    if (rows < 1) return cudaSuccess;
    if (a.topk > 64) return cudaErrorInvalidValue;
    const size_t smem = (size_t)(a.n + 8) * sizeof(float);
    const auto al16 = [](const void* p) { return (((uintptr_t)p) & 15) == 0; };
    const int sms = device_sms();
    if (rows > glue_block_rows(a, sms) && a.n % 64 == 0 && a.n <= 128 * GLUE_PIECES && al16(a.grouped) && al16(a.x_in) && al16(a.y_out) &&
        al16(a.norm_w) && al16(a.router_scale) && al16(a.rin))
        return launch_glue_warps<2>(a, rows, sms, stream);
    if (a.n <= 4096) {
        // every thread owns 4 columns: wide rows and small batches get the largest block
        const int threads = (rows <= 16 || a.n > 1024) ? 1024 : 256;
        return launch_pdl(sum_in_chain(a.n, 1) ? glue_rows_kernel<4, 8, true> : glue_rows_kernel<4, 8, false>, dim3(rows), dim3(threads), smem, stream, a);
    }
    if (a.n <= 8192) return launch_pdl(glue_rows_kernel<16, 2, false>, dim3(rows), dim3(512), smem, stream, a);
    return cudaErrorInvalidValue;
}

cudaError_t launch_rmsnorm(const float* x, const float* weight, float* y, int rows, int n, float eps, int with_scale,
                           int* status, cudaStream_t stream) {
    if (rows < 1) return cudaSuccess;
    const size_t smem = (2 * (size_t)n + 8) * sizeof(float);
    const auto kernel = sum_in_chain(n, 1) ? norm_rows_kernel<0, true> : norm_rows_kernel<0, false>;
    const cudaError_t e = allow_row_smem((const void*)kernel, smem);
    if (e != cudaSuccess) return e;
    kernel<<<rows, 256, smem, stream>>>(x, weight, y, n, eps, with_scale, 0.0f, status);
    return launched();
}

// Threads of a row's top-k: one warp selects, four evaluate the exponentials of up to 128 experts.
constexpr int TOPK_THREADS = 160;

cudaError_t launch_router_input(const float* x, const float* scale, float* out, int rows, int n, float eps,
                                float root, int* status, cudaStream_t stream) {
    if (rows < 1) return cudaSuccess;
    const size_t smem = (2 * (size_t)n + 8) * sizeof(float);
    const auto kernel = sum_in_chain(n, 1) ? norm_rows_kernel<1, true> : norm_rows_kernel<1, false>;
    const cudaError_t e = allow_row_smem((const void*)kernel, smem);
    if (e != cudaSuccess) return e;
    kernel<<<rows, 256, smem, stream>>>(x, scale, out, n, eps, 1, root, status);
    return launched();
}

__global__ void __launch_bounds__(TOPK_THREADS)
router_topk_kernel(const float* __restrict__ logits, const float* __restrict__ per_expert_scale,
                   int32_t* __restrict__ selected, float* __restrict__ weights, int E, int topk, int sort_by_expert,
                   int* status) {
    extern __shared__ __align__(16) float tk_sm[];
    pdl_wait();                    // the logits come from the previous kernel
    pdl_launch_dependents();
    float* sc = tk_sm + topk_scratch_floats(E, topk) - 4;
    const float* lr = logits + (size_t)blockIdx.x * E;
    topk_group(true, [&](int e) { return __ldcg(lr + e); }, per_expert_scale, selected + (size_t)blockIdx.x * topk,
               weights + (size_t)blockIdx.x * topk, E, topk, sort_by_expert, status, tk_sm, sc, threadIdx.x,
               blockDim.x, 1);
}

cudaError_t launch_router_topk(const float* logits, const float* per_expert_scale, int32_t* selected, float* weights,
                               int rows, int E, int topk, int sort_by_expert, int* status, cudaStream_t stream) {
    if (rows < 1) return cudaSuccess;
    if (E < 1 || topk < 1 || (size_t)E + (size_t)topk > 6 * 1024) return cudaErrorInvalidValue;     // 48 KB, counted without overflow
    size_t smem = (size_t)topk_scratch_floats(E, topk) * sizeof(float);
    return launch_pdl(router_topk_kernel, dim3(rows), dim3(TOPK_THREADS), smem, stream, logits, per_expert_scale, selected, weights, E,
                      topk, sort_by_expert, status);
}

// The two projection jobs of grouped rows [g0, g0 + cnt) of expert e.
static __device__ __forceinline__ void write_expert_jobs(const MoePlanArgs& a, int e, int g0, int cnt, int slot) {
    const uint8_t* base = a.pool + (size_t)e * a.expert_stride;
    Q4Job gu;
    gu.vals = base; gu.scales = base + a.value_bytes; gu.biases = base + a.value_bytes + a.group_bytes;
    gu.vals2 = base + a.tensor_bytes; gu.scales2 = gu.vals2 + a.value_bytes;
    gu.biases2 = gu.scales2 + a.group_bytes;
    gu.x = a.x; gu.y = a.chain + (size_t)g0 * a.inter;
    gu.x_rows = a.grouped_to_canonical + g0; gu.x_div = a.topk;
    gu.R = a.inter; gu.C = a.hidden; gu.ntok = cnt; gu.x_stride = a.hidden; gu.y_stride = a.inter;
    a.gateup_jobs[slot] = gu;
    Q4Job dn;
    dn.vals = base + 2 * a.tensor_bytes; dn.scales = dn.vals + a.value_bytes;
    dn.biases = dn.scales + a.group_bytes;
    dn.vals2 = nullptr; dn.scales2 = nullptr; dn.biases2 = nullptr;
    dn.x = a.chain + (size_t)g0 * a.inter; dn.y = a.grouped_out + (size_t)g0 * a.hidden;
    dn.x_rows = nullptr; dn.x_div = 1;
    dn.R = a.hidden; dn.C = a.inter; dn.ntok = cnt; dn.x_stride = a.inter; dn.y_stride = a.hidden;
    a.down_jobs[slot] = dn;
}

// ---- grouping ---------------------------------------------------------------
// Stable counting sort of the selections by expert (src/tensorops.c:239-289,
// src/moe_group.c:83-161): grouped order = expert ascending, then canonical
// index ascending.  One block; the canonical range is cut into 32 contiguous
// segments (one per warp), each warp histograms its segment, a scan over
// (expert, segment) gives every warp its starting slot per expert, and each
// warp then walks its segment in order, ranking equal experts inside a 32-wide
// step with match_any.  Experts outside [expert_begin, expert_end) keep their
// slots in the global order but get no job descriptor.
// NB blocks, a cluster if more than one: each takes a contiguous part of the selections and learns the others' counts through
// distributed shared memory; the first one writes what there is one of.  A lone block is bound by latencies that grow with the
// selections (a load, a match and a store for every 1024 of them): 1999 rows x 8.
template <int NB>
__global__ void __launch_bounds__(1024) moe_plan_kernel(MoePlanArgs a) {
    extern __shared__ __align__(16) int sp[];
    const int E = a.n_experts;
    const int part = NB > 1 ? (int)blockIdx.x : 0;
    pdl_wait();                    // the logits or the selections come from the previous kernel
    pdl_launch_dependents();
    if (a.logits != nullptr) {
        // fused router top-k for small batches: 128 threads per row, up to 8 rows
        float* tk = (float*)(sp + (34 * E + 4));
        const int grp = threadIdx.x >> 7, ltid = threadIdx.x & 127;
        const int per = topk_scratch_floats(E, a.topk);
        float* mine = tk + grp * per;
        const bool active = grp < a.rows;
        const int row = active ? grp : 0;
        const float* lr = a.logits + (size_t)row * E;
        topk_group(active, [&](int e) { return __ldcg(lr + e); }, a.per_expert_scale, a.selected_out + (size_t)row * a.topk,
                   a.weights_out + (size_t)row * a.topk, E, a.topk, 1, a.status, mine, mine + per - 4, ltid, 128, grp + 1);
        __syncthreads();   // selections written by this block are read back below
    }
    int* hist = sp;               // [32][E]
    int* offs = sp + 32 * E;      // [E+1]
    int* act = offs + (E + 1);    // [E] active prefix
    int* own = act + E;           // [E] this block's selections of an expert (NB > 1)
    const int jobs = a.rows * a.topk;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int j0 = NB > 1 ? min(jobs, part * ((jobs + NB - 1) / NB)) : 0, j1 = NB > 1 ? min(jobs, j0 + (jobs + NB - 1) / NB) : jobs;
    const int seg = (j1 - j0 + 31) / 32;
    const int s0 = min(j1, j0 + warp * seg), s1 = min(j1, s0 + seg);
    for (int i = threadIdx.x; i < 32 * E; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    for (int i = s0 + lane; i < s1; i += 32) {
        const int e = a.selected[i];
        if (e < 0 || e >= E) flag(a.status, SB_ERR_INDEX);
        else atomicAdd(&hist[warp * E + e], 1);
    }
    __syncthreads();
    if constexpr (NB > 1) {
        for (int e = threadIdx.x; e < E; e += blockDim.x) {
            int sum = 0;
#pragma unroll 8
            for (int w = 0; w < 32; w++) sum += hist[w * E + e];
            own[e] = sum;
        }
        cooperative_groups::this_cluster().sync();
    }
    // per expert: exclusive scan over segments (of all blocks), total count left in offs[e]
    for (int e = threadIdx.x; e < E; e += blockDim.x) {
        int run = 0, after = 0;
        if constexpr (NB > 1) {
            int theirs[NB];
#pragma unroll
            for (int b = 0; b < NB; b++) theirs[b] = *cooperative_groups::this_cluster().map_shared_rank(own + e, b);
#pragma unroll
            for (int b = 0; b < NB; b++) {
                run += b < part ? theirs[b] : 0;
                after += b > part ? theirs[b] : 0;
            }
        }
        for (int w = 0; w < 32; w++) {
            const int c = hist[w * E + e];
            hist[w * E + e] = run;
            run += c;
        }
        offs[e] = run + after;
    }
    __syncthreads();
    // exclusive scans over experts (E <= 1024 = one expert per thread): group
    // starts, and the compacted index of each local non-empty expert
    {
        __shared__ int warp_cnt[32], warp_act[32], s_max[32];
        const int e = threadIdx.x;
        const int c = e < E ? offs[e] : 0;
        const int local = (e < E && e >= a.expert_begin && e < a.expert_end && c > 0) ? 1 : 0;
        int pc = c, pa = local, mx = local ? c : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int tc = __shfl_up_sync(0xffffffffu, pc, o);
            const int ta = __shfl_up_sync(0xffffffffu, pa, o);
            if (lane >= o) { pc += tc; pa += ta; }
            mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        }
        if (lane == 31) { warp_cnt[warp] = pc; warp_act[warp] = pa; }
        if (lane == 0) s_max[warp] = mx;
        __syncthreads();
        if (warp == 0) {
            int wc = warp_cnt[lane], wa = warp_act[lane], wm = s_max[lane];
            const int tot_c = wc, tot_a = wa;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int tc = __shfl_up_sync(0xffffffffu, wc, o);
                const int ta = __shfl_up_sync(0xffffffffu, wa, o);
                if (lane >= o) { wc += tc; wa += ta; }
                wm = max(wm, __shfl_xor_sync(0xffffffffu, wm, o));
            }
            warp_cnt[lane] = wc - tot_c;     // exclusive prefix of the warp totals
            warp_act[lane] = wa - tot_a;
            if (lane == 31) {
                offs[E] = wc;
                if (part == 0) *a.n_active = wa;
            }
            if (lane == 0 && part == 0) *a.max_group = wm;
        }
        __syncthreads();
        if (e < E) {
            offs[e] = warp_cnt[warp] + pc - c;
            act[e] = local ? warp_act[warp] + pa - 1 : -1;
        }
    }
    __syncthreads();
    if (part == 0)
        for (int e = threadIdx.x; e <= E; e += blockDim.x) a.group_offsets[e] = offs[e];
    // ordered placement
    for (int i0 = s0; i0 < s1; i0 += 32) {
        const int i = i0 + lane;
        const bool live = i < s1;
        int e = live ? a.selected[i] : -1;
        if (e < 0 || e >= E) {
            e = -1;
            if (live) a.canonical_to_grouped[i] = -1;      // no row: what an earlier batch left there is another token's
        }
        const unsigned peers = __match_any_sync(0xffffffffu, e);
        if (e >= 0) {
            const int before = __popc(peers & ((1u << lane) - 1u));
            const int slot = offs[e] + hist[warp * E + e] + before;
            a.grouped_to_canonical[slot] = i;
            a.canonical_to_grouped[i] = slot;
        }
        __syncwarp();
        if (e >= 0 && (peers >> lane) == 1u)  // highest lane of each peer set bumps the running base
            hist[warp * E + e] += __popc(peers);
        __syncwarp();
    }
    if constexpr (NB > 1) {
        cooperative_groups::this_cluster().sync();         // no block leaves while another may read its counts
        if (part != 0) return;
    }
    if (a.fused_done != nullptr && threadIdx.x < FUSED_MAX_JOBS) a.fused_done[threadIdx.x] = 0;
    __syncthreads();               // the placement is complete: the descriptors below reuse its tables
    if (a.pass_tokens > 0) {
        // one job per pass of up to pass_tokens tokens, the largest passes first: their cost is proportional to
        // their tokens, and with whole groups as jobs the SMs that drew the popular experts finished last (B = 64:
        // a third of the SM time idle)
        __shared__ int s_class[32];
        int* first = hist;         // [E] job index of the expert's first full pass
        int* rest = hist + E;      // [E] ... of its last, shorter one
        const int P = a.pass_tokens;   // < 32
        if (threadIdx.x < 32) s_class[threadIdx.x] = 0;
        __syncthreads();
        for (int e = threadIdx.x; e < E; e += blockDim.x)
            if (act[e] >= 0) {
                const int cnt = offs[e + 1] - offs[e];
                if (cnt / P) atomicAdd(&s_class[0], cnt / P);
                if (cnt % P) atomicAdd(&s_class[P - cnt % P], 1);
            }
        __syncthreads();
        if (threadIdx.x == 0) {
            int run = 0;
            for (int k = 0; k < P; k++) { const int c = s_class[k]; s_class[k] = run; run += c; }
            *a.n_active = run;
        }
        __syncthreads();
        for (int e = threadIdx.x; e < E; e += blockDim.x)
            if (act[e] >= 0) {
                const int cnt = offs[e + 1] - offs[e];
                if (cnt / P) first[e] = atomicAdd(&s_class[0], cnt / P);
                if (cnt % P) rest[e] = atomicAdd(&s_class[P - cnt % P], 1);
            }
        __syncthreads();
        for (int e = warp; e < E; e += 32) {
            if (act[e] < 0) continue;
            const int cnt = offs[e + 1] - offs[e];
            for (int p = lane; p * P < cnt; p += 32)
                write_expert_jobs(a, e, offs[e] + p * P, min(P, cnt - p * P), (p + 1) * P <= cnt ? first[e] + p : rest[e]);
        }
        return;
    }
    // job descriptors for the local, non-empty experts (ascending expert order)
    for (int e = threadIdx.x; e < E; e += blockDim.x) {
        const int slot = act[e];
        if (slot < 0) continue;
        const int g0 = offs[e], cnt = offs[e + 1] - offs[e];
        write_expert_jobs(a, e, g0, cnt, slot);
        if (a.fused_jobs != nullptr && slot < FUSED_MAX_JOBS) {
            FusedJob fj;
            for (int k = 0; k < 3; k++) fj.v[k] = a.pool + (size_t)e * a.expert_stride + k * a.tensor_bytes;
            for (int k = 0; k < 3; k++)
                fj.t[k] = (const uint32_t*)(a.fused_tables + ((size_t)e * 6 + 2 * k) * a.group_bytes);
            fj.g0 = g0; fj.lit = a.fused_lit[e];
            a.fused_jobs[slot] = fj;
        }
    }
}

// The same plan for at most 32 selections (decode batches of a few tokens), with the
// router top-k always fused: TOPK_THREADS threads per row run the top-k, then ONE warp places the
// selections (slot = selections with a smaller expert + earlier selections of the same
// expert, which is the stable counting sort) and every thread derives its experts' group
// starts and descriptors by counting over the <= 32 selections.  No histogram, no block
// scans: a handful of barriers instead of a dozen.
__global__ void __launch_bounds__(4 * TOPK_THREADS) moe_plan_small_kernel(MoePlanArgs a) {
    extern __shared__ __align__(16) int sp[];
    const int E = a.n_experts;
    pdl_wait();                    // the logits come from the previous kernel
    pdl_launch_dependents();
    __shared__ int s_sel[32], s_first[32];
    if (a.fused_done != nullptr && threadIdx.x < FUSED_MAX_JOBS) a.fused_done[threadIdx.x] = 0;
    {
        float* tk = (float*)sp;
        const int grp = threadIdx.x / TOPK_THREADS, ltid = threadIdx.x % TOPK_THREADS;
        const int per = topk_scratch_floats(E, a.topk);
        float* mine = tk + grp * per;
        const bool active = grp < a.rows;
        const int row = active ? grp : 0;
        const float* lr = a.logits + (size_t)row * E;
        topk_group(active, [&](int e) { return __ldcg(lr + e); }, a.per_expert_scale, a.selected_out + (size_t)row * a.topk,
                   a.weights_out + (size_t)row * a.topk, E, a.topk, 1, a.status, mine, mine + per - 4, ltid, TOPK_THREADS, grp + 1);
        __syncthreads();   // selections written by this block are read back below
    }
    const int jobs = a.rows * a.topk;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < 32) {
        int e = lane < jobs ? a.selected[lane] : -1;
        if (lane < jobs && (e < 0 || e >= E)) { flag(a.status, SB_ERR_INDEX); e = -1; }
        int before = 0;
        bool first = true;
        for (int j = 0; j < jobs; j++) {
            const int ej = __shfl_sync(0xffffffffu, e, j);
            if (ej >= 0 && (ej < e || (ej == e && j < lane))) before++;
            if (ej == e && j < lane) first = false;
        }
        if (e >= 0) {
            a.grouped_to_canonical[before] = lane;
            a.canonical_to_grouped[lane] = before;
        } else if (lane < jobs) {
            a.canonical_to_grouped[lane] = -1;             // no row: what an earlier batch left there is another token's
        }
        s_sel[lane] = e;
        s_first[lane] = (e >= 0 && first) ? 1 : 0;
    }
    __syncthreads();
    int valid = 0;
    for (int j = 0; j < jobs; j++) valid += s_sel[j] >= 0 ? 1 : 0;
    for (int e = threadIdx.x; e <= E; e += blockDim.x) {
        int lt = 0, eq = 0, slot = 0;
        for (int j = 0; j < jobs; j++) {
            const int ej = s_sel[j];
            if (ej < 0) continue;
            lt += ej < e ? 1 : 0;
            eq += ej == e ? 1 : 0;
            slot += (s_first[j] && ej < e && ej >= a.expert_begin && ej < a.expert_end) ? 1 : 0;
        }
        a.group_offsets[e] = e < E ? lt : valid;
        if (e == E || eq == 0 || e < a.expert_begin || e >= a.expert_end) continue;
        const int g0 = lt, cnt = eq;
        write_expert_jobs(a, e, g0, cnt, slot);
        if (a.fused_jobs != nullptr && slot < FUSED_MAX_JOBS) {
            FusedJob fj;
            for (int k = 0; k < 3; k++) fj.v[k] = a.pool + (size_t)e * a.expert_stride + k * a.tensor_bytes;
            for (int k = 0; k < 3; k++)
                fj.t[k] = (const uint32_t*)(a.fused_tables + ((size_t)e * 6 + 2 * k) * a.group_bytes);
            fj.g0 = g0; fj.lit = a.fused_lit[e];
            a.fused_jobs[slot] = fj;
        }
    }
    if (threadIdx.x == 0) {
        int n_active = 0, max_group = 0;
        for (int j = 0; j < jobs; j++) {
            const int ej = s_sel[j];
            if (!s_first[j] || ej < a.expert_begin || ej >= a.expert_end) continue;
            n_active++;
            int cnt = 0;
            for (int k = 0; k < jobs; k++) cnt += s_sel[k] == ej ? 1 : 0;
            max_group = max(max_group, cnt);
        }
        *a.n_active = n_active;
        *a.max_group = max_group;
    }
}

// One block / a cluster of eight, top-8 (event pairs, us): 128 rows 10.7 / 12.6, 192 rows 12.7 / 12.6, 256 rows 12.7 / 12.7, 384 rows
// 14.7 / 12.7, 512 rows 16.2 / 12.7, 1024 rows 21.2 / 13.4, 1999 rows 33.2 / 14.9.
constexpr int PLAN_BLOCKS = 8;             // the portable cluster size
constexpr long PLAN_CLUSTER_JOBS = 2048;   // selections

cudaError_t launch_moe_plan(const MoePlanArgs& a, cudaStream_t stream) {
    if (a.logits != nullptr && a.rows >= 1 && a.rows <= 4 && a.rows * a.topk <= 32) {
        const size_t small = (size_t)a.rows * topk_scratch_floats(a.n_experts, a.topk) * sizeof(float);
        if (small <= 40 * 1024) {
            return launch_pdl(moe_plan_small_kernel, dim3(1), dim3(TOPK_THREADS * a.rows), small, stream, a);
        }
    }
    size_t smem = (size_t)(34 * a.n_experts + 4) * sizeof(int);
    if (a.logits != nullptr) {
        if (a.rows > 8) return cudaErrorInvalidValue;
        smem += (size_t)8 * topk_scratch_floats(a.n_experts, a.topk) * sizeof(float);
    }
    if (smem > 160 * 1024) return cudaErrorInvalidValue;
    if (a.logits == nullptr && (long)a.rows * a.topk >= PLAN_CLUSTER_JOBS) {
        smem += (size_t)a.n_experts * sizeof(int);
        cudaError_t e = ensure_dynamic_smem((const void*)moe_plan_kernel<PLAN_BLOCKS>, (size_t)(164 * 1024));
        if (e != cudaSuccess) return e;
        return launch_pdl_cluster(moe_plan_kernel<PLAN_BLOCKS>, PLAN_BLOCKS, dim3(1024), smem, stream, a);
    }
    if (smem > PLAIN_DYNAMIC_SMEM) {
        cudaError_t e = ensure_dynamic_smem((const void*)moe_plan_kernel<1>, (size_t)(160 * 1024));
        if (e != cudaSuccess) return e;
    }
    return launch_pdl(moe_plan_kernel<1>, dim3(1), dim3(1024), smem, stream, a);
}

}  // namespace sb
