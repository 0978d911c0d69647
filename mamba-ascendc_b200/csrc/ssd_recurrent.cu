// Short sequences (a generation step of one token, a handful of speculative or streamed tokens): the recurrence itself,
// token by token, with the state in registers,
//
//   S <- exp(A q_t) S + (q_t x_t) B_t^T ;  out_t = (S C_t + D .* x_t) .* silu(z_t)        q_t = clamp(softplus(dt_t + bias))
//
// in one launch, fp32 throughout.  The tile kernels work on 128 tokens at a time, so a call with one token paid for
// 127 of padding, four launches, the framework's padding copies and its element-wise epilogue.
//
// What bounds it: one token moves the state once in each direction and nothing else of size, so it is bound by HBM (and
// by launch latency when the state is small); with more tokens the fp32 pipe takes over.  A row of the state (P index) lies
// along `LPR` lanes, four columns each, and a thread owns four rows, so that its 64 bytes are in flight at
// once and the four dot products with C share their shuffles (halving exchange: 6 instead of 20 for 32 lanes).  CTAs are
// small (128 threads) so that one sequence of a few heads still spreads over the SMs.  Tokens pass through shared
// memory sixteen at a time.  One token of [16, 24, 64, 128] (25 MB of state in and out): 7.0 us = 3.6 TB/s, where the
// padded tile route spent 165 us; [64, 128, 64, 64], 268 MB: 49 us = 5.5 TB/s.
#include "ssd_host.h"
#include "ssd_pdl.cuh"
#include "ssd_tile.cuh"

namespace ssd {

namespace {

constexpr int kRecThreads = 128;
constexpr int kRecRows = 4;     // state rows of one thread
constexpr int kRecTokens = 16;  // tokens staged at a time
constexpr int kRecMaxState = 128;

struct RecArgs {
    const float *x, *dt, *dt_bias, *A, *B, *C, *D, *z, *initial;
    float *out, *final_state;
    int d_mode;
};

// LPR lanes share a row of the state: LPR * 4 >= dstate.
template <int LPR>
__global__ void __launch_bounds__(kRecThreads)
recurrent_kernel(const RecArgs a, const SsdShape s, int row_blocks, int tokens_staged) {
    after_previous();
    allow_next();
    constexpr int kGroups = kRecThreads / LPR;
    constexpr int kCtaRows = kGroups * kRecRows;
    extern __shared__ __align__(16) float rec_smem[];
    const int N = s.dstate, P = s.headdim, H = s.nheads, G = s.ngroups, L = s.seqlen;
    float* sb = rec_smem;                             // [tokens][N]
    float* sc = sb + tokens_staged * N;               // [tokens][N]
    float* sx = sc + tokens_staged * N;               // [tokens][kCtaRows]
    float* sz = sx + tokens_staged * kCtaRows;        // [tokens][kCtaRows], only with z
    float* sq = sz + (a.z != nullptr ? tokens_staged * kCtaRows : 0);  // [tokens] q
    float* sa = sq + tokens_staged;                   // [tokens] exp(A q)

    const int tid = threadIdx.x;
    const int lane = tid % LPR, group = tid / LPR;
    const int pb = blockIdx.x % row_blocks;
    const size_t bh = blockIdx.x / row_blocks;
    const int h = static_cast<int>(bh % H), b = static_cast<int>(bh / H);
    const int g = h / (H / G);
    const int p_first = pb * kCtaRows, p0 = p_first + group * kRecRows;
    const int n0 = lane * 4;
    const bool in_row = n0 < N;

    float4 st[kRecRows];
#pragma unroll
    for (int r = 0; r < kRecRows; ++r) {
        st[r] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (a.initial != nullptr && in_row && p0 + r < P)
            st[r] = __ldcs(reinterpret_cast<const float4*>(a.initial + (bh * P + p0 + r) * N + n0));
    }
    const float decay = a.A[h], bias = a.dt_bias != nullptr ? a.dt_bias[h] : 0.f;
    // after the exchange below this thread holds the dot product of row `my_row` of its group
    const bool upper = (lane & (LPR / 2)) != 0, odd = (lane & (LPR / 4)) != 0;
    const int my_row = (upper ? 2 : 0) + (odd ? 1 : 0);
    const int my_p = p0 + my_row;
    const bool writes = (lane & (LPR / 4 - 1)) == 0 && my_p < P;
    const float d = a.d_mode == 0 || my_p >= P ? 0.f : a.d_mode == 1 ? a.D[h] : a.D[static_cast<size_t>(h) * P + my_p];

    for (int t0 = 0; t0 < L; t0 += tokens_staged) {
        const int nt = min(tokens_staged, L - t0);
        const size_t tok = static_cast<size_t>(b) * L + t0;
        if (t0 > 0) __syncthreads();  // the previous tokens have been used
        for (int i = tid; i < nt * (N / 4); i += kRecThreads) {
            const int t = i / (N / 4), c = (i - t * (N / 4)) * 4;
            const size_t o = ((tok + t) * G + g) * N + c;
            *reinterpret_cast<float4*>(sb + t * N + c) = *reinterpret_cast<const float4*>(a.B + o);
            *reinterpret_cast<float4*>(sc + t * N + c) = *reinterpret_cast<const float4*>(a.C + o);
        }
        for (int i = tid; i < nt * kCtaRows; i += kRecThreads) {
            const int t = i / kCtaRows, r = i % kCtaRows;
            const size_t o = ((tok + t) * H + h) * P + p_first + r;
            const bool in = p_first + r < P;
            sx[i] = in ? a.x[o] : 0.f;
            if (a.z != nullptr) sz[i] = in ? a.z[o] : 0.f;
        }
        if (tid < nt) {
            float w = a.dt[(tok + tid) * H + h] + bias;
            if ((s.flags & SSD_FLAG_DT_SOFTPLUS) != 0) w = softplus_f(w);
            w = fminf(fmaxf(w, s.dt_min), s.dt_max);
            sq[tid] = w;
            sa[tid] = expf(decay * w);
        }
        __syncthreads();
        for (int t = 0; t < nt; ++t) {
            const float al = sa[t], q = sq[t];
            const float4 xv = *reinterpret_cast<const float4*>(sx + t * kCtaRows + group * kRecRows);
            const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 bv = in_row ? *reinterpret_cast<const float4*>(sb + t * N + n0) : zero;
            const float4 cv = in_row ? *reinterpret_cast<const float4*>(sc + t * N + n0) : zero;
            const float qx[kRecRows] = {q * xv.x, q * xv.y, q * xv.z, q * xv.w};
            float v[kRecRows];
#pragma unroll
            for (int r = 0; r < kRecRows; ++r) {
                st[r].x = fmaf(al, st[r].x, qx[r] * bv.x);
                st[r].y = fmaf(al, st[r].y, qx[r] * bv.y);
                st[r].z = fmaf(al, st[r].z, qx[r] * bv.z);
                st[r].w = fmaf(al, st[r].w, qx[r] * bv.w);
                v[r] = fmaf(st[r].x, cv.x, fmaf(st[r].y, cv.y, fmaf(st[r].z, cv.z, st[r].w * cv.w)));
            }
            // four sums over LPR lanes: half the lanes keep rows 0 and 1, the other half 2 and 3, then one row each
            const float r0 = __shfl_xor_sync(0xffffffffu, upper ? v[0] : v[2], LPR / 2);
            const float r1 = __shfl_xor_sync(0xffffffffu, upper ? v[1] : v[3], LPR / 2);
            const float k0 = (upper ? v[2] : v[0]) + r0, k1 = (upper ? v[3] : v[1]) + r1;
            float y = (odd ? k1 : k0) + __shfl_xor_sync(0xffffffffu, odd ? k0 : k1, LPR / 4);
#pragma unroll
            for (int m = LPR / 8; m > 0; m >>= 1) y += __shfl_xor_sync(0xffffffffu, y, m);
            if (writes) {
                const int r = group * kRecRows + my_row;
                float o = y;
                if (a.d_mode != 0) o += sx[t * kCtaRows + r] * d;
                if (a.z != nullptr) {
                    const float zv = sz[t * kCtaRows + r];
                    o *= zv / (1.f + expf(-zv));
                }
                a.out[((tok + t) * H + h) * P + my_p] = o;
            }
        }
    }
    if (a.final_state != nullptr && in_row) {
#pragma unroll
        for (int r = 0; r < kRecRows; ++r)
            if (p0 + r < P) __stcs(reinterpret_cast<float4*>(a.final_state + (bh * P + p0 + r) * N + n0), st[r]);
    }
}

template <int LPR>
int launch_recurrent(const RecArgs& a, const SsdShape& s, cudaStream_t stream) {
    constexpr int kCtaRows = kRecThreads / LPR * kRecRows;
    const int row_blocks = (s.headdim + kCtaRows - 1) / kCtaRows;
    const int64_t blocks = static_cast<int64_t>(s.batch) * s.nheads * row_blocks;
    if (blocks > 0x7fffffff) return SSD_ERR_RANGE;
    const int tokens = s.seqlen < kRecTokens ? s.seqlen : kRecTokens;
    const size_t smem = sizeof(float) * tokens * (2 * s.dstate + (a.z != nullptr ? 2 : 1) * kCtaRows + 2);
    launch_plain(recurrent_kernel<LPR>, static_cast<unsigned>(blocks), kRecThreads, smem, stream, a, s, row_blocks, tokens);
    return launch_status();
}
static_assert(sizeof(float) * kRecTokens * (2 * kRecMaxState + 2 * (kRecThreads / 8 * kRecRows) + 2) <= 48 * 1024,
              "the staged tokens fit the default shared memory");

}  // namespace

}  // namespace ssd

extern "C" int ssd_recurrent_fwd(const SsdShape* shape, const float* x, const float* dt, const float* dt_bias,
                                 const float* A, const float* bm, const float* cm, const float* D, int d_mode,
                                 const float* z, const float* initial_state, float* out, float* final_state,
                                 ssd_stream_t stream) {
    using namespace ssd;
    if (shape == nullptr) return SSD_ERR_NULL;
    const SsdShape& s = *shape;
    if (s.batch <= 0 || s.seqlen <= 0 || s.nheads <= 0 || s.headdim <= 0 || s.dstate <= 0 || s.ngroups <= 0 ||
        s.nheads % s.ngroups != 0 || !(s.dt_min <= s.dt_max) || d_mode < 0 || d_mode > 2)
        return SSD_ERR_SHAPE;
    if (s.dstate % 4 != 0 || s.dstate > kRecMaxState || s.valid_len != 0) return SSD_ERR_UNSUPPORTED;
    if (!x || !dt || !A || !bm || !cm || !out || (d_mode != 0 && !D)) return SSD_ERR_NULL;
    for (const void* p : {static_cast<const void*>(bm), static_cast<const void*>(cm),
                          static_cast<const void*>(initial_state), static_cast<const void*>(final_state)})
        if ((reinterpret_cast<uintptr_t>(p) & 15u) != 0) return SSD_ERR_ALIGN;
    const RecArgs a{x, dt, dt_bias, A, bm, cm, D, z, initial_state, out, final_state, d_mode};
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (s.dstate <= 32) return launch_recurrent<8>(a, s, st);
    if (s.dstate <= 64) return launch_recurrent<16>(a, s, st);
    return launch_recurrent<32>(a, s, st);
}
