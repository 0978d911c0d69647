// D skip connection and SiLU(z) gate around the SSD output, as one pass forward and one pass backward:
//
//   out = (y + D .* x) .* silu(z)                 (ssd_reference.py:300-318; either of D, z may be absent)
//
//   dy  = dout .* silu(z) ;  dz = dout .* (y + D .* x) .* silu'(z) ;  dD = sum dy .* x
//   (dx += D .* dy happens in the epilogue of the dx kernel, ssd_bwd_dx.cu)
//
// The reference fuses these into its state-epilogue and gate kernels (mamba2_ssd_state_epilogue.cpp:413-482,
// bwd_gate/design.md:8-13).  Element-wise and bandwidth bound: the tensors are walked as [tokens, H*P] with
// float4 accesses along the row; dD is reduced in two phases in a fixed order (fp64 in the second phase).
//
// What bounds these kernels is how many loads are in flight, so both dimensions of a CTA follow the shape: `ct`
// threads along a row and `rt` rows side by side (a row of a few hundred channels otherwise leaves most of
// the CTA idle), kGateUnroll rows per thread at once, and row blocks small enough to give every SM several CTAs.
#include "ssd_host.h"
#include "ssd_pdl.cuh"

namespace ssd {

namespace {

constexpr int kGateThreads = 256;
constexpr int kGateUnroll = 4;        // rows of one thread in flight together
constexpr int kGateMaxRows = 128;     // tokens per CTA in the backward pass at most: their products are summed in fp32 ...
constexpr int kGateCtasWanted = 1184; // ... fewer when that leaves less than eight CTAs per SM of 148, ...
constexpr int kGateMinRows = 32;      // ... but there not so few that adding up the partials takes longer than forming them

// How [rows, cols / 4] float4s are laid over CTAs: `colblocks` blocks of `ct` threads along a row, `rt` rows side by
// side in a CTA.  ct * rt <= kGateThreads, and ct is as even a share of the row as the block count allows.  Row blocks fill
// grid.y and, beyond 65535, grid.z, so that any number of rows keeps its blocks of at most kGateMaxRows.
struct GateGrid {
    int ct, rt, colblocks, rows_per_cta;
    long long rowblocks;
    dim3 grid() const {
        const long long slices = (rowblocks + 65534) / 65535;
        return dim3(colblocks, static_cast<unsigned>(slices == 1 ? rowblocks : 65535), static_cast<unsigned>(slices));
    }
};
GateGrid gate_grid(long long rows, int cols, int min_rows) {
    GateGrid g;
    const int c4 = cols / 4;
    g.colblocks = (c4 + kGateThreads - 1) / kGateThreads;
    g.ct = (c4 + g.colblocks - 1) / g.colblocks;
    g.rt = kGateThreads / g.ct < kGateMaxRows / kGateUnroll ? kGateThreads / g.ct : kGateMaxRows / kGateUnroll;
    const int least = g.rt * kGateUnroll > min_rows ? g.rt * kGateUnroll : min_rows;
    g.rows_per_cta = kGateMaxRows;
    while (g.rows_per_cta / 2 >= least && (rows + g.rows_per_cta - 1) / g.rows_per_cta * g.colblocks < kGateCtasWanted)
        g.rows_per_cta /= 2;
    g.rowblocks = (rows + g.rows_per_cta - 1) / g.rows_per_cta;
    return g;
}

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ float sigmoidf_(float v) { return 1.f / (1.f + expf(-v)); }

// D for the four columns c..c+3 of a row (c % 4 == 0): d_mode 0 none, 1 per head [H], 2 per channel [H,P].
__device__ __forceinline__ float4 load_d(const float* D, int d_mode, int c, int p_dim) {
    if (d_mode == 2) return ld4(D + c);
    if (d_mode == 1) {
        const float d = D[c / p_dim];
        return make_float4(d, d, d, d);
    }
    return make_float4(0.f, 0.f, 0.f, 0.f);
}

template <bool HAS_D, bool HAS_Z>
__global__ void __launch_bounds__(kGateThreads)
gate_skip_fwd_kernel(const float* __restrict__ y, const float* __restrict__ x, const float* __restrict__ D, int d_mode,
                     const float* __restrict__ z, float* __restrict__ out, long long rows, int cols, int p_dim, int ct,
                     int rt, int rows_per_cta) {
    after_previous();
    allow_next();
    const int tx = threadIdx.x % ct, ty = threadIdx.x / ct;
    const long long row_block = static_cast<long long>(blockIdx.z) * gridDim.y + blockIdx.y;
    const int c = (blockIdx.x * ct + tx) * 4;
    if (c >= cols || ty >= rt) return;
    const float4 d = load_d(D, d_mode, c, p_dim);
    const long long r0 = row_block * rows_per_cta;
    const long long r1 = r0 + rows_per_cta < rows ? r0 + rows_per_cta : rows;
    for (long long r = r0 + ty; r < r1; r += kGateUnroll * rt) {
        float4 v[kGateUnroll], xv[kGateUnroll], zv[kGateUnroll];
#pragma unroll
        for (int u = 0; u < kGateUnroll; ++u) {
            const long long ru = r + u * rt;
            if (ru < r1) {
                const size_t o = static_cast<size_t>(ru) * cols + c;
                v[u] = ld4(y + o);
                if (HAS_D) xv[u] = ld4(x + o);
                if (HAS_Z) zv[u] = ld4(z + o);
            }
        }
#pragma unroll
        for (int u = 0; u < kGateUnroll; ++u) {
            const long long ru = r + u * rt;
            if (ru >= r1) break;
            if (HAS_D) {
                v[u].x += d.x * xv[u].x;
                v[u].y += d.y * xv[u].y;
                v[u].z += d.z * xv[u].z;
                v[u].w += d.w * xv[u].w;
            }
            if (HAS_Z) {
                v[u].x *= zv[u].x * sigmoidf_(zv[u].x);
                v[u].y *= zv[u].y * sigmoidf_(zv[u].y);
                v[u].z *= zv[u].z * sigmoidf_(zv[u].z);
                v[u].w *= zv[u].w * sigmoidf_(zv[u].w);
            }
            st4(out + static_cast<size_t>(ru) * cols + c, v[u]);
        }
    }
}

// Backward.  dy and dz are written only with z (without, dy equals dout and the caller uses dout itself).
// part[row_block][cols] receives this CTA's sum over its tokens of dy .* x: each thread over its own rows, then the
// `rt` rows that stand side by side in order.
template <bool HAS_D, bool HAS_Z>
__global__ void __launch_bounds__(kGateThreads)
gate_skip_bwd_kernel(const float* __restrict__ dout, const float* __restrict__ y, const float* __restrict__ x,
                     const float* __restrict__ D, int d_mode, const float* __restrict__ z, float* __restrict__ dy,
                     float* __restrict__ dz, float* __restrict__ part, long long rows, int cols, int p_dim, int ct, int rt,
                     int rows_per_cta) {
    after_previous();
    allow_next();
    __shared__ float4 sums[kGateThreads];
    const int tx = threadIdx.x % ct, ty = threadIdx.x / ct;
    const long long row_block = static_cast<long long>(blockIdx.z) * gridDim.y + blockIdx.y;
    const int c = (blockIdx.x * ct + tx) * 4;
    const bool active = c < cols && ty < rt && row_block * rows_per_cta < rows;
    const long long r0 = row_block * rows_per_cta;
    const long long r1 = r0 + rows_per_cta < rows ? r0 + rows_per_cta : rows;
    constexpr int kUnroll = HAS_Z ? 2 : kGateUnroll;  // four tensors a row with z: eight float4 in flight
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (active) {
        const float4 d = load_d(D, d_mode, c, p_dim);
        for (long long r = r0 + ty; r < r1; r += kUnroll * rt) {
            float4 g[kUnroll], xv[kUnroll], zv[kUnroll], yv[kUnroll];
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) {
                const long long ru = r + u * rt;
                if (ru < r1) {
                    const size_t o = static_cast<size_t>(ru) * cols + c;
                    g[u] = ld4(dout + o);
                    xv[u] = HAS_D ? ld4(x + o) : make_float4(0.f, 0.f, 0.f, 0.f);
                    if (HAS_Z) {
                        zv[u] = ld4(z + o);
                        yv[u] = ld4(y + o);
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) {
                const long long ru = r + u * rt;
                if (ru >= r1) break;
                float4 gy = g[u];
                if (HAS_Z) {
                    const size_t o = static_cast<size_t>(ru) * cols + c;
                    const float zz[4] = {zv[u].x, zv[u].y, zv[u].z, zv[u].w};
                    const float pre[4] = {yv[u].x + d.x * xv[u].x, yv[u].y + d.y * xv[u].y, yv[u].z + d.z * xv[u].z,
                                          yv[u].w + d.w * xv[u].w};
                    const float gg[4] = {gy.x, gy.y, gy.z, gy.w};
                    float oy[4], oz[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float s = sigmoidf_(zz[i]);
                        oy[i] = gg[i] * zz[i] * s;
                        oz[i] = gg[i] * pre[i] * s * (1.f + zz[i] * (1.f - s));
                    }
                    gy = make_float4(oy[0], oy[1], oy[2], oy[3]);
                    st4(dy + o, gy);
                    st4(dz + o, make_float4(oz[0], oz[1], oz[2], oz[3]));
                }
                acc.x += gy.x * xv[u].x;
                acc.y += gy.y * xv[u].y;
                acc.z += gy.z * xv[u].z;
                acc.w += gy.w * xv[u].w;
            }
        }
    }
    if (!HAS_D) return;
    sums[threadIdx.x] = acc;
    __syncthreads();
    if (active && ty == 0) {
        for (int i = 1; i < rt; ++i) {
            const float4 o = sums[i * ct + tx];
            acc.x += o.x;
            acc.y += o.y;
            acc.z += o.z;
            acc.w += o.w;
        }
        st4(part + static_cast<size_t>(row_block) * cols + c, acc);
    }
}

// Second phase of dD: a CTA per head, `lanes` threads per channel that take the row blocks in turn; their fp64 sums
// are added in order, then (per-head D) the channels.
__global__ void gate_dd_reduce_kernel(const float* __restrict__ part, int row_blocks, int cols, int p_dim, int d_mode,
                                      int lanes, float* __restrict__ dD) {
    after_previous();
    allow_next();
    extern __shared__ double red[];
    const int h = blockIdx.x, p = threadIdx.x % p_dim, l = threadIdx.x / p_dim;
    double s = 0.0;
    if (l < lanes)
#pragma unroll 8
        for (int rb = l; rb < row_blocks; rb += lanes) s += part[static_cast<size_t>(rb) * cols + h * p_dim + p];
    red[threadIdx.x] = s;
    __syncthreads();
    if (l == 0) {
        for (int i = 1; i < lanes; ++i) s += red[i * p_dim + p];
        if (d_mode == 2) dD[h * p_dim + p] = static_cast<float>(s);
    }
    if (d_mode == 2) return;
    __syncthreads();
    if (l == 0) red[p] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        double t = 0.0;
        for (int i = threadIdx.x; i < p_dim; i += 32) t += red[i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (threadIdx.x == 0) dD[h] = static_cast<float>(t);
    }
}

// The tensors as rows of `cols` values, `heads` times `p` of them (of D): with SSD_FLAG_EXTENTS the caller's tokens, and the
// parts of a head together.
struct GateDims {
    long long rows;
    int cols, heads, p;
};
int gate_dims(const SsdShape* s, GateDims* d) {
    if (!s) return SSD_ERR_NULL;
    if (s->batch <= 0 || s->seqlen <= 0 || s->nheads <= 0 || s->headdim <= 0) return SSD_ERR_SHAPE;
    const int parts = head_parts(*s), tokens = row_tokens(*s);
    if (s->nheads % parts != 0 || tokens > s->seqlen) return SSD_ERR_SHAPE;
    if (s->headdim % 4 != 0 || s->headdim * static_cast<long long>(parts) > 1024) return SSD_ERR_UNSUPPORTED;
    *d = GateDims{static_cast<long long>(s->batch) * tokens, s->nheads * s->headdim, s->nheads / parts, s->headdim * parts};
    return SSD_OK;
}

}  // namespace

}  // namespace ssd

extern "C" size_t ssd_gate_partial_floats(const SsdShape* shape) {
    ssd::GateDims n;
    if (ssd::gate_dims(shape, &n) != SSD_OK) return 0;
    return static_cast<size_t>(ssd::gate_grid(n.rows, n.cols, ssd::kGateMinRows).rowblocks) * n.cols;
}

extern "C" int ssd_gate_skip_fwd(const SsdShape* shape, const float* y, const float* x, const float* D, int d_mode,
                                 const float* z, float* out, ssd_stream_t stream) {
    using namespace ssd;
    GateDims n;
    const int rc = gate_dims(shape, &n);
    if (rc != SSD_OK) return rc;
    if (!y || !out || (d_mode != 0 && (!D || !x))) return SSD_ERR_NULL;
    if (d_mode < 0 || d_mode > 2) return SSD_ERR_SHAPE;
    if (!aligned16(y, x, z, out, d_mode == 2 ? D : nullptr)) return SSD_ERR_ALIGN;
    const GateGrid g = gate_grid(n.rows, n.cols, 1);
    auto launch = [&](auto kernel) {
        launch_plain(kernel, g.grid(), kGateThreads, 0,
                     reinterpret_cast<cudaStream_t>(stream), y, x, D, d_mode, z, out, n.rows, n.cols, n.p, g.ct, g.rt,
                     g.rows_per_cta);
    };
    if (d_mode != 0)
        z ? launch(gate_skip_fwd_kernel<true, true>) : launch(gate_skip_fwd_kernel<true, false>);
    else
        z ? launch(gate_skip_fwd_kernel<false, true>) : launch(gate_skip_fwd_kernel<false, false>);
    return launch_status();
}

extern "C" int ssd_gate_skip_bwd(const SsdShape* shape, const float* dout, const float* y, const float* x, const float* D,
                                 int d_mode, const float* z, float* dy, float* dz, float* dD_partial, float* dD,
                                 ssd_stream_t stream) {
    using namespace ssd;
    GateDims n;
    const int rc = gate_dims(shape, &n);
    if (rc != SSD_OK) return rc;
    if (d_mode < 0 || d_mode > 2) return SSD_ERR_SHAPE;
    if (!dout || (z && (!y || !dy || !dz)) || (d_mode != 0 && (!D || !x || !dD_partial || !dD))) return SSD_ERR_NULL;
    if (!z && d_mode == 0) return SSD_OK;  // nothing to do
    if (!aligned16(dout, y, x, z, dy, dz, dD_partial, d_mode == 2 ? D : nullptr)) return SSD_ERR_ALIGN;
    const GateGrid g = gate_grid(n.rows, n.cols, kGateMinRows);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    auto launch = [&](auto kernel) {
        launch_plain(kernel, g.grid(), kGateThreads, 0, st, dout, y, x, D, d_mode, z,
                     dy, dz, dD_partial, n.rows, n.cols, n.p, g.ct, g.rt, g.rows_per_cta);
    };
    if (d_mode != 0)
        z ? launch(gate_skip_bwd_kernel<true, true>) : launch(gate_skip_bwd_kernel<true, false>);
    else
        launch(gate_skip_bwd_kernel<false, true>);
    if (d_mode != 0) {
        const int lanes = 1024 / n.p;
        const int threads = (lanes * n.p + 31) / 32 * 32;
        launch_plain(gate_dd_reduce_kernel, n.heads, threads, threads * sizeof(double), st, dD_partial,
                     static_cast<int>(g.rowblocks), n.cols, n.p, d_mode, lanes, dD);
    }
    return launch_status();
}
