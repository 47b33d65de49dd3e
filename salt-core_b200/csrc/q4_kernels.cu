// Grouped affine-Q4 projections: the choice of kernel, and the one that takes any C and any byte alignment with
// absolute group indices (rows may straddle quantisation groups), one warp per (row, token).  It reproduces the
// reference row DAG (src/kernels.c:220-250) bit for bit, like batch_kernel for the aligned shapes.
#include "internal.h"
#include "pdl.cuh"
#include "q4_core.cuh"

namespace sb {

// Any shape, any alignment.  Lane l owns accumulator l (columns c == l mod 32).
template <int NMAT>
__global__ void __launch_bounds__(128)
q4_generic_kernel(const Q4Job* __restrict__ jobs, const int* __restrict__ njobs_dev) {
    const int job_id = blockIdx.z;
    if (njobs_dev != nullptr && job_id >= *njobs_dev) return;
    const Q4Job jb = jobs[job_id];
    const int r = blockIdx.x * 4 + (threadIdx.x >> 5);
    const int tok = blockIdx.y;
    if (r >= jb.R || tok >= jb.ntok) return;
    const int lane = threadIdx.x & 31;
    const int xrow = jb.x_rows ? (jb.x_rows[tok] / jb.x_div) : tok;
    const float* x = jb.x + (size_t)xrow * jb.x_stride;
    float yv[NMAT];
#pragma unroll
    for (int m = 0; m < NMAT; m++) {
        const uint8_t* vals = m == 0 ? jb.vals : jb.vals2;
        const uint8_t* scales = m == 0 ? jb.scales : jb.scales2;
        const uint8_t* biases = m == 0 ? jb.biases : jb.biases2;
        float acc = 0.0f;
        for (int c = lane; c < jb.C; c += 32) {
            const size_t k = (size_t)r * (size_t)jb.C + (size_t)c;
            const size_t g = k >> 6;
            const uint8_t byte = vals[k >> 1];
            const uint32_t q = (k & 1) ? (uint32_t)(byte >> 4) : (uint32_t)(byte & 15u);
            const uint32_t hs = (uint32_t)scales[2 * g] | ((uint32_t)scales[2 * g + 1] << 8);
            const uint32_t hb = biases ? ((uint32_t)biases[2 * g] | ((uint32_t)biases[2 * g + 1] << 8)) : 0u;
            float d = __fmul_rn((float)q, bf16_bits_to_f32(hs));
            d = __fadd_rn(d, bf16_bits_to_f32(hb));
            acc = __fadd_rn(acc, __fmul_rn(d, x[c]));
        }
        // L_j for j = lane & 3 is needed in lanes 0..3: gather acc[j + 4a] in order.
        float L = 0.0f;
#pragma unroll
        for (int a = 0; a < 8; a++) L = __fadd_rn(L, __shfl_sync(0xffffffffu, acc, (lane & 3) + 4 * a));
        const float L2 = __shfl_sync(0xffffffffu, L, 2);
        const float L1 = __shfl_sync(0xffffffffu, L, 1);
        const float L3 = __shfl_sync(0xffffffffu, L, 3);
        yv[m] = __fadd_rn(__fadd_rn(L, L2), __fadd_rn(L1, L3));  // meaningful in lane 0
    }
    if (lane == 0) {
        float* yrow = jb.y + (size_t)tok * jb.y_stride;
        yrow[r] = (NMAT == 2) ? __fmul_rn(gelu_tanh_exact(yv[0]), yv[NMAT - 1]) : yv[0];
    }
}

bool q4_stores_lines(int C, int nmat, bool aligned) { return aligned && q4_batch_supported(C, nmat); }

cudaError_t launch_q4_jobs(const Q4Job* jobs, int njobs_max, const int* njobs_dev, int max_rows, int max_tok, int C,
                           int nmat, bool aligned, cudaStream_t stream, int pdl, bool alone) {
    if (njobs_max < 1 || max_rows < 1 || max_tok < 1) return cudaSuccess;
    if (q4_stores_lines(C, nmat, aligned))
        return launch_q4_batch(jobs, njobs_max, njobs_dev, max_rows, max_tok, C, nmat, stream, pdl, alone);
    dim3 grid((max_rows + 3) / 4, max_tok, njobs_max);
    if (grid.y > 65535 || grid.z > 65535) return cudaErrorInvalidValue;
    if (nmat == 2) q4_generic_kernel<2><<<grid, 128, 0, stream>>>(jobs, njobs_dev);
    else q4_generic_kernel<1><<<grid, 128, 0, stream>>>(jobs, njobs_dev);
    return launched();
}

}  // namespace sb
