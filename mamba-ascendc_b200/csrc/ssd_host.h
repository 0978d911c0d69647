// Host-side helpers shared by the launchers: error codes, the shape record,
// tensor-map construction for fp32 tiles and launch-error translation.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <utility>

#include "../../include/ssd_b200.h"

namespace ssd {

// ---- what the caller's tensors and the internal buffers look like (see SSD_FLAG_EXTENTS)
inline __host__ __device__ bool has_extents(const SsdShape& s) { return (s.flags & SSD_FLAG_EXTENTS) != 0; }
// tokens per sequence of the token-major tensors
inline __host__ __device__ int row_tokens(const SsdShape& s) {
    return has_extents(s) && s.valid_len > 0 ? s.valid_len : s.seqlen;
}
// heads of the kernels per head of dt, A, dt_bias and D[H]
inline __host__ __device__ int head_parts(const SsdShape& s) {
    return has_extents(s) ? static_cast<int>((s.flags >> 8) & 0xFFFFu) + 1 : 1;
}
constexpr int kStateRows = 64;  // headdim of the internal state buffers
inline __host__ __device__ int state_cols(const SsdShape& s) { return s.dstate <= 64 ? 64 : 128; }

// Tensor map over fp32 data for TMA tile loads with 128-byte swizzle.
// dims/box are innermost first; strides_bytes has rank-1 entries (stride of
// dims[1], dims[2], ...).  The innermost box extent must be 32 floats.
// A map depends only on the base address and the geometry, so encoded maps are kept in a small
// process-wide table and reused by later calls on the same buffers (a training loop whose allocator hands
// out the same blocks every step never encodes again).
int make_tmap_f32(CUtensorMap* map, const void* base, int rank, const uint64_t* dims, const uint64_t* strides_bytes,
                  const uint32_t* box);

// 2-D row-major fp32 matrix [rows x cols], box = [box_rows x 32].
inline int make_tmap_f32_2d(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows) {
    const uint64_t dims[2] = {cols, rows};
    const uint64_t strides[1] = {cols * sizeof(float)};
    const uint32_t box[2] = {32u, box_rows};
    return make_tmap_f32(map, base, 2, dims, strides, box);
}

// Token-major activation [batch, tokens, heads, width] (x, dout, out: width = P; B, C: heads = G, width = N); box = 32
// floats of one head for 128 tokens.  Batch is a dimension of its own, so that a tile that runs over the end of a
// sequence is filled with zeros (load) or cut off (store) instead of reaching into the next one.
inline int make_tmap_f32_tokens(CUtensorMap* map, const void* base, const SsdShape& s, uint64_t heads, uint64_t width) {
    const uint64_t tokens = row_tokens(s), row = width * sizeof(float);
    const uint64_t dims[4] = {width, heads, tokens, static_cast<uint64_t>(s.batch)};
    const uint64_t strides[3] = {row, heads * row, tokens * heads * row};
    const uint32_t box[4] = {32u, 1u, 128u, 1u};
    return make_tmap_f32(map, base, 4, dims, strides, box);
}
// The state buffers [B,H,K,64,N'] as rows; box = 32 floats of 64 rows.
inline int make_tmap_f32_states(CUtensorMap* map, const void* base, const SsdShape& s) {
    const uint64_t rows = static_cast<uint64_t>(s.batch) * s.nheads * (s.seqlen / s.tile) * kStateRows;
    return make_tmap_f32_2d(map, base, rows, state_cols(s), 64);
}

// Index of the current device, or -1.
int current_device();

// SMs of the current device (the grid size of the persistent kernels); 0 on error.  Looked up once per device.
int sm_count();

// Raise a kernel's dynamic shared-memory limit once per device (the attribute belongs to the function in
// each device's context); `done` is the launcher's own bit set, one bit per device.
int set_max_smem_once(const void* func, size_t bytes, std::atomic<uint64_t>& done);

// Into how many work items the heads of a group are dealt, for a kernel whose `items` = batch * ngroups * tiles work
// items take `slots` CTAs at a time.  An item treats `unit` heads at once and costs `overhead_halves` half units besides
// (its B and C tiles and their product); a round costs as much as one item.  Few groups and a short sequence leave SMs
// without an item, and a split gives them one at the price of the overhead: 8192 tokens of 32 heads in one group (64 items
// on 148 SMs) take 44 instead of 75 us in the output kernel and 27 instead of 64 us in the state kernel, with two and
// four items per group.  A split has to promise 5% to be taken.
int choose_head_split(int64_t items, int heads_per_group, int slots, int unit, int overhead_halves);

// Kernel launches.  Chained: programmatic stream order -- the kernel may start while the one before it in the stream is
// still running its last CTAs, and waits (after_previous, ssd_pdl.cuh) before it touches global memory, so that its start-up
// (launch, barriers, tensor memory) lies under the tail of that kernel.  For kernels that fill an SM with one CTA (launch_tiles):
// forward of [4,2048,16,64,128] 82.4 -> 77.7 us, its training step 258 -> 251 us, Vision network 2571 -> 2493 us, no difference at
// [8,4096,32,64,64] (14 work items per SM), 1% slower at [8,4096,256,64,64] (110 per SM), where it is left out.  Not for kernels
// of small CTAs (launch_plain): placed early, they pile up on the SMs that are free first and stay there (with all
// kernels chained, prefill went from 137 to 145 us and the training step at [8,4096,32] from 1027 to 1052).
template <class... Expected, class... Args>
inline void launch_config(bool chained, void (*kernel)(Expected...), dim3 grid, unsigned block, size_t smem,
                          cudaStream_t stream, Args&&... args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = dim3(block);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    config.attrs = &attr;
    config.numAttrs = chained ? 1 : 0;
    (void)cudaLaunchKernelEx(&config, kernel, static_cast<Expected>(args)...);  // launch_status() picks an error up
}
constexpr int kChainedItemsPerSm = 32;
template <class Kernel, class... Args>
inline void launch_tiles(int64_t items, Kernel kernel, dim3 grid, unsigned block, size_t smem, cudaStream_t stream,
                         Args&&... args) {
    launch_config(items <= int64_t(kChainedItemsPerSm) * sm_count(), kernel, grid, block, smem, stream,
                  std::forward<Args>(args)...);
}
template <class Kernel, class... Args>
inline void launch_plain(Kernel kernel, dim3 grid, unsigned block, size_t smem, cudaStream_t stream, Args&&... args) {
    launch_config(false, kernel, grid, block, smem, stream, std::forward<Args>(args)...);
}

// Whether every pointer (null ones aside) takes 16-byte accesses.
template <class... P>
inline bool aligned16(const P*... p) {
    return ((reinterpret_cast<uintptr_t>(p) | ...) & 15u) == 0;
}

inline int launch_status() {
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? SSD_OK : SSD_ERR_LAUNCH;
}

}  // namespace ssd
