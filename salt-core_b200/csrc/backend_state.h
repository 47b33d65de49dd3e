// Process-wide state of the salt_gpu_* backend (one calling thread at a time,
// as the reference surface assumes).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <unordered_map>
#include <vector>

#include "../../include/salt_gpu_b200.h"

namespace sb {

struct Q4Job;

// Fixed capacities, allocated once by salt_gpu_init and never grown by an
// operation: 2048 tokens x top-8 rows of 2816 floats per staging buffer.
constexpr size_t SB_STAGE_FLOATS = (size_t)16384 * 2816;
constexpr uint32_t SB_MAX_JOBS = 16384;

struct Resource {
    uint32_t kind = 0, id = 0;
    const uint8_t* host = nullptr;
    size_t nbytes = 0;
    uint8_t* dev = nullptr;
    bool active = false;
    int policy = 0;
    uint64_t window_off = 0, window_bytes = 0;
};

struct Tensor {
    uint32_t kind = 0, id = 0;
    int bits = 0, R = 0, C = 0;      // bits: 4 = affine Q4, 104 = NVFP4
    uint64_t voff = 0, soff = 0, boff = 0, aoff = 0;
    size_t vbytes = 0, gbytes = 0;
    const uint8_t *dv = nullptr, *ds = nullptr, *db = nullptr;  // device views (16-byte aligned)
    float weight_divisor = 0.0f, input_global = 0.0f;           // NVFP4 per-tensor scalars
    std::vector<void*> owned;                                   // private aligned copies
};

struct Selected {
    bool active = false;
    uint64_t logical_id = 0;
    const void* base = nullptr;
    const void* payload = nullptr;
    size_t nbytes = 0;
    uint8_t* dev = nullptr;          // where the payload lives in HBM: `own`, or a residency seat
    uint8_t* own = nullptr;          // allocation of the copying bind, kept for the slot's next occupant
    size_t own_cap = 0;
    bool resident = false;           // bound by salt_gpu_selected_resource_bind_resident
    uint64_t generation = 0;
};

struct Backend {
    bool ready = false;
    int mapped_only = 0, defer = 0;
    std::vector<Resource> resources;
    std::unordered_map<const void*, Tensor> tensors;
    std::unordered_map<const void*, Tensor> arena;
    std::vector<Selected> selected;
    std::vector<int> logical_to_slot;
    bool selected_fenced = false;
    SaltGpuBatchStatsV2 stats = {};
    uint64_t copied_bytes = 0, peak_window = 0;
    cudaStream_t stream = nullptr;
    // One upload block each in pinned host memory and in HBM: descriptors, then activations (x).  A synchronous call
    // puts its descriptors right before x, so that one copy takes both; the descriptors of asynchronous calls fill
    // the block from its start (d_jobs, h_jobs).
    uint8_t *d_up = nullptr, *h_up = nullptr;
    float *d_x = nullptr, *d_y = nullptr, *d_mid = nullptr;
    float *h_x = nullptr, *h_y = nullptr;
    float* hd_y = nullptr;             // h_y as the device sees it
    Q4Job *d_jobs = nullptr, *h_jobs = nullptr;
    int *d_status = nullptr, *h_status = nullptr;   // one word of mapped host memory: written by kernels that fail only
    size_t stage_floats = 0, job_cap = 0, x_cursor = 0, job_cursor = 0;
    bool in_flight = false;            // asynchronous calls since the last synchronisation
};

// Results up to these sizes are written straight into pinned host memory by the kernel, larger ones are copied afterwards.
// A kernel whose stores leave as whole lines (batch_kernels.cu, bf16 batches) gains 2 us at 16 KB and 10 at 128 KB (32768
// rows of 256 columns: 37 -> 27 us; 1000 rows x 100 tokens, 390 KB, is the first shape where it loses, 68 against 71).  One
// float per block or warp (q8, any-shape Q4 and NVFP4) or four (bf16 matvec) are as many separate writes over the bus: direct
// is 1 to 7 us faster at 16 KB, between 2 us slower and 4 us faster at 32 to 64 KB from host to host, and far slower above
// (any-shape Q4, 131072 rows of 72: 179 to 207 us against 89).
constexpr size_t SB_DIRECT_LINES = (size_t)512 * 1024, SB_DIRECT_FLOATS = (size_t)32 * 1024;

extern Backend g_backend;
bool cuda_ok(cudaError_t e, const char* what);
bool stream_fence();                   // waits for asynchronous calls, if there were any
// Uploads `head` bytes of descriptors (already at (uint8_t*)h_x - head) and `bytes` of activations in one copy.
bool stage_upload(size_t head, size_t bytes, const char* what);
// Where a call's kernels put `bytes` of results (whole_lines: how they store them), and the end of the call: the results that
// were put at y_dev are in h_y, the stream is idle.
float* stage_out(size_t bytes, bool whole_lines);
bool stage_finish(const float* y_dev, size_t bytes, const char* what);
uint64_t launch_count();
uintptr_t residency_seat_address(int seat, size_t nbytes);
void residency_shutdown();

}  // namespace sb
