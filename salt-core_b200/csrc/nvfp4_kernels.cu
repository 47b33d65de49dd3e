// NVFP4 (E2M1 codes, one E4M3FN scale per 16 elements, per-tensor fp32 scalars)
// kernels, bit-exact against the reference src/nvfp4.c:
//
//   nvfp4_qdq_kernel     dynamic group-16 activation quantise -> dequantise
//                        (salt_nvfp4_quantize_input_reference, nvfp4.c:82-130)
//   nvfp4_generic_kernel W4A4 projection on the dequantised activations with the canonical
//                        32-accumulator order (nvfp4.c:173-192, 157-171), any C that is a
//                        multiple of 16; multiples of 256 take batch_kernels.cu
//
// The encoders are arithmetic instead of the reference's nearest-code searches:
// "nearest, ties to the even code" over a monotone code table is round-to-
// nearest-even in that format (checked against the searches in the tests).
#include <algorithm>

#include "fp4_core.cuh"
#include "internal.h"
#include "pdl.cuh"
#include "q4_core.cuh"

namespace sb {

static __device__ __forceinline__ void flag_status(int* status, int bit) {
    if (status) atomicOr(status, bit);
}

// E4M3FN encode of a finite value in [0, 448] (nvfp4.c:41-63): nearest code,
// ties to the even code.
__device__ __forceinline__ uint32_t e4m3_encode_pos(float v) {
    if (v < 0.015625f) return (uint32_t)__float2int_rn(__fmul_rn(v, 512.0f));  // subnormal grid 2^-9
    uint32_t b = __float_as_uint(v);
    b = (b + 0x7ffffu + ((b >> 20) & 1u)) >> 20;   // round to 3 mantissa bits, ties to even
    return (((b >> 3) - 120u) << 3) | (b & 7u);
}

// E2M1 encode of a value already clamped to [-6, 6] (nvfp4.c:65-80): magnitudes
// {0, .5, 1, 1.5, 2, 3, 4, 6}; on a tie the even code wins.
__device__ __forceinline__ uint32_t e2m1_encode(float t) {
    const float m = fabsf(t);
    uint32_t c = (m > 0.25f) + (m >= 0.75f) + (m > 1.25f) + (m >= 1.75f) + (m > 2.5f) + (m >= 3.5f) + (m > 5.0f);
    if (__float_as_uint(t) & 0x80000000u) c |= 8u;
    return c;
}

// E2M1 decode (nvfp4.c:19-23): both zero codes give +0.
__device__ __forceinline__ float e2m1_decode(uint32_t code) {
    const uint32_t e = (code >> 1) & 3u, m = code & 1u;
    float v = e == 0 ? (m ? 0.5f : 0.0f) : __uint_as_float(((e + 126u) << 23) | (m << 22));
    if (v == 0.0f) return 0.0f;
    return (code & 8u) ? -v : v;
}

// One thread per block of 16 activations.  ig_rows[row] is the row's input
// global scale.  Non-finite activations set the status word (the reference
// function returns -1).
// src_rows != null: row r of the call reads activation row src_rows[r % src_mod] / src_div (the grouped
// order of a MoE layer: several quantisations of the same token row with different global scales).
// GEGLU: the activations are formed on the fly as gelu_tanh(x[i]) * up[i] (reference gemma4.c:80-83 and the
// product of gemma4_text.c:8927-8930) - the quantiser of a layer's second projection batch needs no GeGLU buffer.
template <bool WANT_DQ, bool GEGLU>
__global__ void __launch_bounds__(512)
nvfp4_qdq_kernel(const float* __restrict__ x, const float* __restrict__ up, int rows, int C,
                 const float* __restrict__ ig_rows, uint8_t* __restrict__ packed, uint8_t* __restrict__ scales,
                 float* __restrict__ dequant, int* status, const int* __restrict__ src_rows, int src_mod, int src_div) {
    // blocks (x, y): row x, 16-element blocks y * blockDim.x + thread; the row's source and scale are found once
    pdl_wait();                    // scales, row table and activations come from the kernels before this one
    pdl_launch_dependents();
    const int bpr = C >> 4;
    const int row = blockIdx.x;
    const float ig = ig_rows[row];
    if (!(ig > 0.0f)) return;         // a row nobody will read (its expert lives on another rank): its source may be unwritten
    const int in_row = src_rows ? src_rows[row % src_mod] / src_div : row;
    for (int blk = blockIdx.y * blockDim.x + threadIdx.x; blk < bpr; blk += gridDim.y * blockDim.x) {
        const float4* in4 = (const float4*)(x + (size_t)in_row * C + blk * 16);
        float v[16];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float4 t = in4[i];
            v[4 * i] = t.x; v[4 * i + 1] = t.y; v[4 * i + 2] = t.z; v[4 * i + 3] = t.w;
        }
        if (GEGLU) {
            const float4* up4 = (const float4*)(up + (size_t)in_row * C + blk * 16);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float4 t = up4[i];
                v[4 * i] = __fmul_rn(gelu_tanh_exact(v[4 * i]), t.x);
                v[4 * i + 1] = __fmul_rn(gelu_tanh_exact(v[4 * i + 1]), t.y);
                v[4 * i + 2] = __fmul_rn(gelu_tanh_exact(v[4 * i + 2]), t.z);
                v[4 * i + 3] = __fmul_rn(gelu_tanh_exact(v[4 * i + 3]), t.w);
            }
        }
        float amax = 0.0f;
        bool bad = false;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const float m = fabsf(v[i]);
            bad |= !finite_f(m);
            if (m > amax) amax = m;
        }
        if (bad) {
            flag_status(status, SB_ERR_NONFINITE);
            continue;
        }
        float raw = __fmul_rn(ig, __fmul_rn(amax, 0.16666667163372039794921875f));
        if (raw > 448.0f) raw = 448.0f;
        const uint32_t sc = e4m3_encode_pos(raw);
        const float scale = e4m3_decode(sc);
        const float out_scale = scale == 0.0f ? 0.0f : __fdiv_rn(ig, scale);
        const float dq_scale = WANT_DQ ? __fdiv_rn(scale, ig) : 0.0f;
        uint32_t lo = 0, hi = 0;
        float dq[16];
#pragma unroll
        for (int i = 0; i < 16; i++) {
            float t = __fmul_rn(v[i], out_scale);
            if (t > 6.0f) t = 6.0f;
            if (t < -6.0f) t = -6.0f;
            const uint32_t c = e2m1_encode(t);
            if (WANT_DQ) dq[i] = __fmul_rn(e2m1_decode(c), dq_scale);
            if (i < 8) lo |= c << (4 * i);
            else hi |= c << (4 * (i - 8));
        }
        scales[(size_t)row * bpr + blk] = (uint8_t)sc;
        *(uint2*)(packed + (size_t)row * (C >> 1) + blk * 8) = make_uint2(lo, hi);
        if (WANT_DQ) {
            float4* out4 = (float4*)(dequant + (size_t)row * C + blk * 16);
#pragma unroll
            for (int i = 0; i < 4; i++) out4[i] = make_float4(dq[4 * i], dq[4 * i + 1], dq[4 * i + 2], dq[4 * i + 3]);
        }
    }
}

cudaError_t launch_nvfp4_qdq(const float* x, int rows, int C, const float* ig_rows, uint8_t* packed, uint8_t* scales,
                             float* dequant, int* status, cudaStream_t stream, const int* src_rows, int src_mod,
                             int src_div, const float* geglu_up) {
    if (rows < 1) return cudaSuccess;
    if (src_rows && (src_mod < 1 || src_div < 1 || geglu_up)) return cudaErrorInvalidValue;
    const int bpr = C >> 4;
    const int threads = bpr >= 512 ? 512 : ((bpr + 31) & ~31);
    const dim3 grid((unsigned)rows, (unsigned)std::min(65535, (bpr + threads - 1) / threads));
#define SB_QDQ(DQ, GG) \
    launch_pdl(nvfp4_qdq_kernel<DQ, GG>, grid, dim3(threads), 0, stream, x, geglu_up, rows, C, ig_rows, packed, scales, \
               dequant, status, src_rows, src_mod, src_div)
    if (dequant) return geglu_up ? SB_QDQ(true, true) : SB_QDQ(true, false);
    return geglu_up ? SB_QDQ(false, true) : SB_QDQ(false, false);     // the tensor-core consumer reads codes and scales only
#undef SB_QDQ
}

// Any C (multiple of 16), any alignment: one warp per (row, token), lane l owns
// accumulator l.
__global__ void __launch_bounds__(128)
nvfp4_generic_kernel(const Fp4Job* __restrict__ jobs, const int* __restrict__ njobs_dev) {
    if (njobs_dev != nullptr && (int)blockIdx.z >= *njobs_dev) return;
    const Fp4Job jb = jobs[blockIdx.z];
    const int r = blockIdx.x * 4 + (threadIdx.x >> 5), tok = blockIdx.y;
    if (r >= jb.R || tok >= jb.ntok) return;
    const int lane = threadIdx.x & 31;
    const float* x = jb.x + (size_t)tok * jb.x_stride;
    float acc = 0.0f;
    for (int c = lane; c < jb.C; c += 32) {
        const size_t k = (size_t)r * jb.C + c;
        const uint8_t byte = jb.codes[k >> 1];
        const uint32_t code = (k & 1) ? (byte >> 4) : (byte & 15u);
        const float sc = __fmul_rn(e4m3_decode(jb.scales[(size_t)r * (jb.C >> 4) + (c >> 4)]), jb.wg);
        const float w = __fmul_rn(e2m1_decode(code), sc);
        acc = __fadd_rn(acc, __fmul_rn(w, x[c]));
    }
    float L = 0.0f;
#pragma unroll
    for (int a = 0; a < 8; a++) L = __fadd_rn(L, __shfl_sync(0xffffffffu, acc, (lane & 3) + 4 * a));
    const float L2 = __shfl_sync(0xffffffffu, L, 2);
    const float L1 = __shfl_sync(0xffffffffu, L, 1);
    const float L3 = __shfl_sync(0xffffffffu, L, 3);
    if (lane == 0) jb.y[(size_t)tok * jb.y_stride + r] = __fadd_rn(__fadd_rn(L, L2), __fadd_rn(L1, L3));
}

// ---- a MoE layer of NVFP4 experts (reference caller: models/gemma4-26b-a4b/src/gemma4_text.c:8912-8945,
// two projection batches with the GeGLU between them) ------------------------------------------------
// The input global scale of every grouped row (gate rows [0, J), up rows [J, 2J) of the gathered activations; down rows
// [0, J)), and the projection jobs: one per pass of up to pass_tokens tokens of an expert, the largest passes first (gate and
// up of pass i are gu_jobs[2 i] and [2 i + 1]), with their number; or, for the tensor cores, the jobs of whole groups.
// (One job per expert in grids as deep as the batch left three of four blocks empty at 16 tokens and 180 000 of 196 000 at
// 256, each with its shared memory until it had read its job.)
// A thread per expert.  The kernel is a link of a decode layer's chain of launches, so everything that does not depend on the
// routing is read before the wait and the slots need one barrier: a class' base is the sum of the counts before it.
__global__ void __launch_bounds__(1024) nvfp4_moe_plan_kernel(Fp4PlanArgs a) {
    constexpr int P = Q4_PASS_TOKENS;
    __shared__ int s_count[P], s_next[P];         // passes by size, largest first; those that have a slot
    const int E = a.n_experts, e = threadIdx.x;
    const bool local = e >= a.expert_begin && e < a.expert_end;
    Fp4ExpertDesc d;
    if (local) d = a.experts[e - a.expert_begin];
    if (threadIdx.x < P) s_count[threadIdx.x] = s_next[threadIdx.x] = 0;
    __syncthreads();
    pdl_wait();                    // the group offsets come from the plan kernel before this one
    pdl_launch_dependents();
    const int g0 = e < E ? a.group_offsets[e] : 0, cnt = e < E ? a.group_offsets[e + 1] - g0 : 0;
    // rows past the last group (selections without an expert) are skipped by the quantiser too: their entries of the row
    // table are an earlier batch's and may lie past this one's rows
    for (int r = a.group_offsets[E] + (int)threadIdx.x; r < a.rows; r += blockDim.x)
        a.ig_gu[r] = a.ig_gu[a.rows + r] = a.ig_dn[r] = 0.0f;
    // pass_tokens = 0: groups are not cut, and come in any order
    const int nfull = a.pass_tokens ? cnt / P : 0, rest = a.pass_tokens ? cnt % P : cnt, k_rest = a.pass_tokens ? (P - rest) % P : 0;
    const bool jobs = a.gu_jobs != nullptr && local && cnt > 0;
    if (jobs) {
        if (nfull) atomicAdd(&s_count[0], nfull);
        if (rest) atomicAdd(&s_count[k_rest], 1);
    }
    __syncthreads();
    if (threadIdx.x == 0 && a.gu_jobs != nullptr) {
        int run = 0;
        for (int k = 0; k < P; k++) run += s_count[k];
        a.n_jobs[0] = 2 * run;
        a.n_jobs[1] = run;
    }
    if (e < E) {
        if (jobs) {
            const int first = nfull ? atomicAdd(&s_next[0], nfull) : 0;
            int last = rest ? atomicAdd(&s_next[k_rest], 1) : 0;
            for (int k = 0; k < k_rest; k++) last += s_count[k];
            for (int p = 0; p < nfull + (rest ? 1 : 0); p++) {
                const int slot = p < nfull ? first + p : last;
                const size_t row = (size_t)g0 + (size_t)p * P;
                Fp4Job j;
                j.ntok = p < nfull ? P : rest;
                j.R = a.inter; j.C = a.hidden; j.x_stride = a.hidden; j.y_stride = a.inter;
                j.codes = d.codes[0]; j.scales = d.scales[0]; j.wg = d.wg[0];
                j.x = a.dq_gu + row * a.hidden; j.y = a.gate_out + row * a.inter;
                a.gu_jobs[2 * slot] = j;
                j.codes = d.codes[1]; j.scales = d.scales[1]; j.wg = d.wg[1];
                j.x = a.dq_gu + (row + a.rows) * a.hidden; j.y = a.up_out + row * a.inter;
                a.gu_jobs[2 * slot + 1] = j;
                j.R = a.hidden; j.C = a.inter; j.x_stride = a.inter; j.y_stride = a.hidden;
                j.codes = d.codes[2]; j.scales = d.scales[2]; j.wg = d.wg[2];
                j.x = a.dq_dn + row * a.inter; j.y = a.grouped_out + row * a.hidden;
                a.dn_jobs[slot] = j;
            }
        }
        if (a.tc_gu != nullptr) {
            // the up matrix follows the gate codes (M rows) and the gate scales (M / 8 rows of H / 2 bytes) in the expert's
            // slot; the quantised activations' block scales use the rows of the packed codes (gate [0, J), up [J, 2J);
            // down [0, J) after the second quantisation); scale rows are C / 16 bytes long: in those units the up scales
            // start 9 M rows (one tensor) after the gate scales
            const int M = a.inter;
            Fp4TcJob t;
            t.ntok = local ? cnt : 0; t.w_slice = local ? e - a.expert_begin : 0;
            t.R = M; t.y_stride = M; t.w_row0 = 0; t.ws_row0 = 0; t.x_row0 = g0;
            t.wg = local ? d.wg[0] : 0.0f; t.ig = local ? d.ig[0] : 1.0f; t.y = a.gate_out + (size_t)g0 * M;
            a.tc_gu[e] = t;
            t.w_row0 = M + (M >> 3); t.ws_row0 = 9 * M; t.x_row0 = a.rows + g0;
            t.wg = local ? d.wg[1] : 0.0f; t.ig = local ? d.ig[1] : 1.0f; t.y = a.up_out + (size_t)g0 * M;
            a.tc_gu[E + e] = t;
            t.R = a.hidden; t.y_stride = a.hidden; t.w_row0 = 0; t.ws_row0 = 0; t.x_row0 = g0;
            t.wg = local ? d.wg[2] : 0.0f; t.ig = local ? d.ig[2] : 1.0f; t.y = a.grouped_out + (size_t)g0 * a.hidden;
            a.tc_dn[e] = t;
        }
        for (int t = 0; t < cnt; t++) {               // rows of remote experts are marked (scale 0) and skipped by the quantiser
            a.ig_gu[g0 + t] = local ? d.ig[0] : 0.0f;
            a.ig_gu[a.rows + g0 + t] = local ? d.ig[1] : 0.0f;
            a.ig_dn[g0 + t] = local ? d.ig[2] : 0.0f;
        }
    }
}

cudaError_t launch_nvfp4_moe_plan(const Fp4PlanArgs& a, cudaStream_t stream) {
    if ((a.pass_tokens != 0 && a.pass_tokens != Q4_PASS_TOKENS) || a.n_experts < 1 || a.n_experts > 1024) return cudaErrorInvalidValue;
    return launch_pdl(nvfp4_moe_plan_kernel, dim3(1), dim3((a.n_experts + 31) & ~31), 0, stream, a);
}

cudaError_t launch_nvfp4_jobs(const Fp4Job* jobs, int njobs, int max_rows, int max_tok, int C, bool aligned,
                              cudaStream_t stream, const int* njobs_dev) {
    if (njobs < 1 || max_rows < 1 || max_tok < 1) return cudaSuccess;
    if (aligned && fp4_batch_supported(C)) return launch_fp4_batch(jobs, njobs, njobs_dev, max_rows, max_tok, C, stream);
    dim3 grid((max_rows + 3) / 4, max_tok, njobs);
    if (grid.y > 65535 || grid.z > 65535) return cudaErrorInvalidValue;
    nvfp4_generic_kernel<<<grid, 128, 0, stream>>>(jobs, njobs_dev);
    return launched();
}

}  // namespace sb
