// Element-wise companions of the SSD inside a Mamba-2 block, forward only, for the Vision-Mamba2 network of
// benchmark configuration 4 (RMSNorm -> in_proj -> depthwise causal conv1d + SiLU -> SSD -> gated RMSNorm ->
// out_proj).  Bandwidth-bound kernels that each read their input once and write their output once, in place of
// the ten-odd framework launches per step they replace:
//
//   block_rmsnorm_kernel     out = x * rsqrt(mean(x^2) + eps) * w,  optionally x <- (x + D .* s) * silu(z) first (the SSD's
//                            skip connection and the gated norm)
//   block_conv_silu_kernel   depthwise causal convolution of width 4 along the sequence, bias, SiLU, and the split of
//                            the result into contiguous x [B,L,d_in], B [B,L,GN] and C [B,L,GN] tensors; on the way dt
//                            [B,L,H] from the columns behind them and A = -exp(A_log)
//
// Inputs may be column slices of a wider row-major matrix (the in_proj output holds z | xBC | dt side by side),
// hence the explicit row strides; rows need not be 16-byte aligned, so loads are scalar (or of two floats where rows are
// 8-byte aligned) with lanes along the channels (coalesced).  The reference's demo network applies the same operations with framework calls
// (mamba_torch/vmamba2_network.py:197-302).
#include "ssd_host.h"
#include "ssd_pdl.cuh"

namespace ssd {

namespace {

__device__ __forceinline__ float silu_f(float v) { return v / (1.f + expf(-v)); }

// One warp per row, VEC = 2 floats (1 where rows are not 8-byte aligned) per lane at a time, ITERS of them, all loads of the
// row in flight together.  Bound by HBM: 384 channels with gate and skip at 16384 rows (101 MB) 19 us = 5.3 TB/s; with scalar
// loads and a fixed sixteen guarded steps the norm alone took 17 us on 25 MB, now 5.3 us.
constexpr int kMaxRow = 512;

struct NormArgs {
    const float *x, *z, *skip, *d, *w;
    float* out;
    long long x_stride, z_stride, rows;
    int dim, headdim;
    float eps;
};

template <int VEC, int ITERS, bool GATE, bool SKIP>
__global__ void __launch_bounds__(256)
block_rmsnorm_kernel(const NormArgs a) {
    after_previous();
    allow_next();
    const int lane = threadIdx.x & 31;
    const long long row = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= a.rows) return;
    float v[ITERS][VEC], zv[ITERS][VEC], sv[ITERS][VEC];
    auto load = [&](float* dst, const float* src) {
        if constexpr (VEC == 2) {
            const float2 f = *reinterpret_cast<const float2*>(src);
            dst[0] = f.x;
            dst[1] = f.y;
        } else {
            dst[0] = *src;
        }
    };
#pragma unroll
    for (int i = 0; i < ITERS; ++i) {
        const int c = (lane + 32 * i) * VEC;
#pragma unroll
        for (int j = 0; j < VEC; ++j) v[i][j] = 0.f;
        if (c < a.dim) {
            load(v[i], a.x + row * a.x_stride + c);
            if (GATE) load(zv[i], a.z + row * a.z_stride + c);
            if (SKIP) load(sv[i], a.skip + row * a.dim + c);
        }
    }
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < ITERS; ++i) {
        const int c = (lane + 32 * i) * VEC;
        if (c < a.dim) {
            const float d = SKIP ? a.d[c / a.headdim] : 0.f;  // VEC divides headdim: one head per load
#pragma unroll
            for (int j = 0; j < VEC; ++j) {
                if (SKIP) v[i][j] += sv[i][j] * d;
                if (GATE) v[i][j] *= silu_f(zv[i][j]);
                ss = fmaf(v[i][j], v[i][j], ss);
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float r = rsqrtf(ss / static_cast<float>(a.dim) + a.eps);
    float* orow = a.out + row * a.dim;
#pragma unroll
    for (int i = 0; i < ITERS; ++i) {
        const int c = (lane + 32 * i) * VEC;
        if (c < a.dim) {
            float wv[VEC];
            load(wv, a.w + c);
            if constexpr (VEC == 2)
                *reinterpret_cast<float2*>(orow + c) = make_float2(v[i][0] * r * wv[0], v[i][1] * r * wv[1]);
            else
                orow[c] = v[i][0] * r * wv[0];
        }
    }
}

template <int VEC, int ITERS>
int launch_norm(const NormArgs& a, cudaStream_t stream) {
    const long long blocks = (a.rows + 7) / 8;
    if (blocks > 0x7fffffffLL) return SSD_ERR_RANGE;
    auto launch = [&](auto kernel) { launch_plain(kernel, static_cast<unsigned>(blocks), 256, 0, stream, a); };
    if (a.skip != nullptr)
        a.z ? launch(block_rmsnorm_kernel<VEC, ITERS, true, true>) : launch(block_rmsnorm_kernel<VEC, ITERS, false, true>);
    else
        a.z ? launch(block_rmsnorm_kernel<VEC, ITERS, true, false>) : launch(block_rmsnorm_kernel<VEC, ITERS, false, false>);
    return launch_status();
}

// CTA = 128 channels x kConvTokens tokens of one batch row; a thread has its channel's kConvTokens inputs and the three
// before them in flight at once.  Bound by HBM through the loads in flight: 512 channels of [4, 4096] tokens (67 MB)
// 20 us = 3.4 TB/s; 64 tokens per thread with eight loads in flight took 33 us.  weight [C,4] (tap k multiplies the input 3-k tokens
// back), bias [C].  Channels behind the convolved ones are dt: copied as they are.
constexpr int kConvTokens = 16;
constexpr int kGridY = 65535;

struct ConvArgs {
    const float *xbc, *weight, *bias, *a_log;
    float *x_out, *b_out, *c_out, *dt_out, *a_out;
    long long row_stride;
    int seqlen, d_in, gn, heads;  // heads: of dt and A, 0 = neither
};

// SLICED: a sequence of more than 65535 blocks of tokens, the most that grid.y holds, is several slices of grid.z.
template <bool SLICED>
__global__ void __launch_bounds__(128)
block_conv_silu_kernel(const ConvArgs a, int slices) {
    after_previous();
    allow_next();
    const int channels = a.d_in + 2 * a.gn;
    const int c = blockIdx.x * 128 + threadIdx.x;
    if (c >= channels + a.heads) return;
    const long long b = SLICED ? blockIdx.z / slices : blockIdx.z;
    const int t0 = (SLICED ? blockIdx.z % slices * kGridY + blockIdx.y : blockIdx.y) * kConvTokens;
    if (SLICED && t0 >= a.seqlen) return;
    const float* src = a.xbc + (b * a.seqlen) * a.row_stride + c;
    float in[kConvTokens + 3];  // inputs from three tokens back on
#pragma unroll
    for (int i = 0; i < kConvTokens + 3; ++i) {
        const int t = t0 + i - 3;
        in[i] = t >= 0 && t < a.seqlen ? src[t * a.row_stride] : 0.f;
    }
    float* dst;
    int width, col;
    if (c < a.d_in) {
        dst = a.x_out, width = a.d_in, col = c;
    } else if (c < a.d_in + a.gn) {
        dst = a.b_out, width = a.gn, col = c - a.d_in;
    } else if (c < channels) {
        dst = a.c_out, width = a.gn, col = c - a.d_in - a.gn;
    } else {
        dst = a.dt_out, width = a.heads, col = c - channels;
        if (blockIdx.y == 0 && blockIdx.z == 0) a.a_out[col] = -expf(a.a_log[col]);
    }
    dst += (b * a.seqlen) * width + col;
    const int n = min(kConvTokens, a.seqlen - t0);
    if (c >= channels) {
#pragma unroll
        for (int i = 0; i < kConvTokens; ++i)
            if (i < n) dst[static_cast<long long>(t0 + i) * width] = in[i + 3];
        return;
    }
    const float w0 = a.weight[c * 4], w1 = a.weight[c * 4 + 1], w2 = a.weight[c * 4 + 2], w3 = a.weight[c * 4 + 3];
    const float bs = a.bias ? a.bias[c] : 0.f;
#pragma unroll
    for (int i = 0; i < kConvTokens; ++i) {
        const float v = fmaf(w0, in[i], fmaf(w1, in[i + 1], fmaf(w2, in[i + 2], fmaf(w3, in[i + 3], bs))));
        if (i < n) dst[static_cast<long long>(t0 + i) * width] = silu_f(v);
    }
}

}  // namespace

}  // namespace ssd

extern "C" int ssd_block_skip_rmsnorm_fwd(const float* x, long long x_stride, const float* skip, const float* D, int headdim,
                                          const float* z, long long z_stride, const float* w, float* out, long long rows,
                                          int d, float eps, ssd_stream_t stream) {
    using namespace ssd;
    if (!x || !w || !out || (skip && !D)) return SSD_ERR_NULL;
    if (rows <= 0 || d <= 0 || x_stride < d || (z && z_stride < d) || (skip && headdim <= 0)) return SSD_ERR_SHAPE;
    if (d > kMaxRow) return SSD_ERR_UNSUPPORTED;
    const NormArgs a{x, z, skip, D, w, out, x_stride, z_stride, rows, d, headdim, eps};
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const uintptr_t low = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(z) | reinterpret_cast<uintptr_t>(skip) |
                          reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(out);
    const bool pairs = (low & 7u) == 0 && d % 2 == 0 && x_stride % 2 == 0 && (!z || z_stride % 2 == 0) &&
                       (!skip || headdim % 2 == 0);
    if (!pairs) return launch_norm<1, kMaxRow / 32>(a, st);
    if (d <= 192) return launch_norm<2, 3>(a, st);
    if (d <= 384) return launch_norm<2, 6>(a, st);
    return launch_norm<2, kMaxRow / 64>(a, st);
}

extern "C" int ssd_block_rmsnorm_fwd(const float* x, long long x_stride, const float* z, long long z_stride,
                                     const float* w, float* out, long long rows, int d, float eps,
                                     ssd_stream_t stream) {
    return ssd_block_skip_rmsnorm_fwd(x, x_stride, nullptr, nullptr, 0, z, z_stride, w, out, rows, d, eps, stream);
}

extern "C" int ssd_block_conv_split_fwd(const float* xbc, long long row_stride, const float* weight, const float* bias,
                                        const float* a_log, float* x_out, float* b_out, float* c_out, float* dt_out,
                                        float* a_out, int batch, int seqlen, int d_in, int gn, int heads,
                                        ssd_stream_t stream) {
    using namespace ssd;
    if (!xbc || !weight || !x_out || !b_out || !c_out || (heads > 0 && (!a_log || !dt_out || !a_out))) return SSD_ERR_NULL;
    if (batch <= 0 || seqlen <= 0 || d_in <= 0 || gn <= 0 || heads < 0 || row_stride < d_in + 2 * gn + heads)
        return SSD_ERR_SHAPE;
    const long long token_blocks = (static_cast<long long>(seqlen) + kConvTokens - 1) / kConvTokens;
    const int slices = static_cast<int>((token_blocks + kGridY - 1) / kGridY);
    if (batch > 65535 / slices || seqlen > 0x7fffffff - 2 * kConvTokens * kGridY) return SSD_ERR_RANGE;
    const ConvArgs a{xbc, weight, bias, a_log, x_out, b_out, c_out, dt_out, a_out, row_stride, seqlen, d_in, gn, heads};
    const dim3 grid((d_in + 2 * gn + heads + 127) / 128, static_cast<unsigned>(slices == 1 ? token_blocks : kGridY), batch * slices);
    launch_plain(slices == 1 ? block_conv_silu_kernel<false> : block_conv_silu_kernel<true>, grid, 128, 0,
                 reinterpret_cast<cudaStream_t>(stream), a, slices);
    return launch_status();
}

extern "C" int ssd_block_conv_silu_fwd(const float* xbc, long long row_stride, const float* weight, const float* bias,
                                       float* x_out, float* b_out, float* c_out, int batch, int seqlen, int d_in, int gn,
                                       ssd_stream_t stream) {
    return ssd_block_conv_split_fwd(xbc, row_stride, weight, bias, nullptr, x_out, b_out, c_out, nullptr, nullptr, batch,
                                    seqlen, d_in, gn, 0, stream);
}
