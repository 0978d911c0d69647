// Bandwidth-bound scan kernels of the SSD path (no tensor cores):
//   dt_cumsum_kernel        q = softplus(dt), cs = in-tile inclusive cumsum of A*q   (warp scan)
//   state_walk              S_{k+1} = exp(cs_last,k) * S_k + U_k, in place over the chunk states, or the reverse recurrence
//   state_passing_bwd       reverse recurrence, in place over the local dS, with d(cs_last) as well
//   dt_finalize             [B,H,L] -> [B,L,H] transpose of ddt, fixed-order reductions of dA and d(dt_bias)
#include "ssd_host.h"
#include "ssd_pdl.cuh"
#include "ssd_tile.cuh"

namespace ssd {

namespace {

// ------------------------------------------------------------------ dt softplus + cumsum
// CTA = (tile k, block of up to 32 heads, batch b).  The [128 tokens x heads] patch of dt is read with lanes along
// heads (contiguous in memory; with fewer than 32 heads a warp takes several tokens), turned in shared memory, and
// each warp scans its heads with lanes along tokens, four tokens per lane plus a shuffle scan of the lane totals.
// The kernel moves little and is bound by latency: all of a thread's up to 16 loads are in flight before the first
// is used (one load at a time: 5.8 us for a single CTA, 12 us at [8,4096,32]).
__global__ void __launch_bounds__(256)
dt_cumsum_kernel(const float* __restrict__ dt, const float* __restrict__ dt_bias, const float* __restrict__ A,
                 float* __restrict__ q, float* __restrict__ cs, SsdShape s, int head_bits) {
    after_previous();
    allow_next();
    __shared__ float patch[kTile][33];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int k = blockIdx.x, h0 = blockIdx.y * 32, b = blockIdx.z;
    const int heads = min(32, s.nheads - h0);  // <= 1 << head_bits
    const int parts = head_parts(s), tokens = row_tokens(s) - k * kTile;  // tokens of dt from this tile on
    const bool softplus = (s.flags & SSD_FLAG_DT_SOFTPLUS) != 0;
    {
        const int hh = tid & ((1 << head_bits) - 1), t_first = tid >> head_bits, t_step = 256 >> head_bits;
        if (hh < heads) {
            const int source = (h0 + hh) / parts, sources = s.nheads / parts;
            const float bias = dt_bias != nullptr ? dt_bias[source] : 0.f;
            const float* src = dt + (static_cast<size_t>(b) * row_tokens(s) + k * kTile) * sources + source;
            float v[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int t = t_first + i * t_step;
                v[i] = t < kTile && t < tokens ? src[static_cast<size_t>(t) * sources] : 0.f;
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int t = t_first + i * t_step;
                if (t >= kTile) break;
                float w = v[i] + bias;
                if (softplus) w = softplus_f(w);
                w = fminf(fmaxf(w, s.dt_min), s.dt_max);
                if (s.valid_len > 0 && k * kTile + t >= s.valid_len) w = 0.f;  // padding: no step, no decay
                patch[t][hh] = w;
            }
        }
    }
    __syncthreads();
    for (int hh = warp; hh < heads; hh += 8) {
        const int head = h0 + hh;
        const float a = A[head / parts];
        float qv[4], c[4];
        float run = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            qv[i] = patch[lane * 4 + i][hh];
            run += a * qv[i];
            c[i] = run;
        }
        float incl = run;  // inclusive scan of the lane totals
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const float up = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += up;
        }
        const float before = incl - run;
        const size_t o = (static_cast<size_t>(b) * s.nheads + head) * s.seqlen + k * kTile + lane * 4;
        *reinterpret_cast<float4*>(q + o) = make_float4(qv[0], qv[1], qv[2], qv[3]);
        *reinterpret_cast<float4*>(cs + o) = make_float4(before + c[0], before + c[1], before + c[2], before + c[3]);
    }
}

// ------------------------------------------------------------------ state passing, either direction
// One thread owns four consecutive state elements of one (b,h) and walks the tiles, ascending (forward: the buffer holds
// U_k on entry and S_k, the state at the START of tile k, on exit) or descending (backward: dS_k on entry, dU_k on exit);
// the recurrence is the same:  v = states[k] ; states[k] = st ; st = exp(cs_last,k) * st + v.  `end` receives the last st.
//
// Bound by HBM, and by the loads in flight where there are few (b,h) chains to walk: kWalkTiles tiles are requested ahead of
// the kWalkTiles being worked on, and CTAs are small so that few chains still reach every SM.  32 chains of 64 tiles
// (67 MB): 9.8 us = 6.8 TB/s partly from L2, against 26 us with one load ahead and CTAs of 256; 256 chains of 32 tiles (268 MB): 40.2
// us = 6.7 TB/s, against 52.
constexpr int kWalkTiles = 8;
constexpr int kWalkThreads = 64;
template <bool REVERSE>
__global__ void __launch_bounds__(kWalkThreads)
state_walk_kernel(float* __restrict__ states, const float* __restrict__ cs, const float* __restrict__ start,
                  float* __restrict__ end, int nchunks, int n4, int seqlen, int headdim, int dstate4, size_t total) {
    after_previous();
    allow_next();
    const size_t idx = static_cast<size_t>(blockIdx.x) * kWalkThreads + threadIdx.x;
    if (idx >= total) return;
    const int pn4 = kStateRows * n4;
    const size_t bh = idx / pn4;
    const int e = static_cast<int>(idx % pn4);
    const int row = e / n4, col = e % n4;  // of the state; `start` and `end` are [headdim, dstate4]
    const bool inside = row < headdim && col < dstate4;
    const size_t edge = (bh * headdim + row) * dstate4 + col;
    float4* p = reinterpret_cast<float4*>(states) + bh * nchunks * pn4 + e;
    const float* csl = cs + bh * seqlen + (kTile - 1);
    auto tile_of = [&](int i) { return static_cast<size_t>(REVERSE ? nchunks - 1 - i : i); };
    float4 st = start && inside ? reinterpret_cast<const float4*>(start)[edge] : make_float4(0.f, 0.f, 0.f, 0.f);
    float4 u[kWalkTiles];
    float c[kWalkTiles];
#pragma unroll
    for (int i = 0; i < kWalkTiles; ++i)
        if (i < nchunks) {
            u[i] = p[tile_of(i) * pn4];
            c[i] = csl[tile_of(i) * kTile];
        }
    for (int k = 0; k < nchunks; k += kWalkTiles) {
        float4 un[kWalkTiles];
        float cn[kWalkTiles];
#pragma unroll
        for (int i = 0; i < kWalkTiles; ++i)
            if (k + kWalkTiles + i < nchunks) {
                un[i] = p[tile_of(k + kWalkTiles + i) * pn4];
                cn[i] = csl[tile_of(k + kWalkTiles + i) * kTile];
            }
#pragma unroll
        for (int i = 0; i < kWalkTiles; ++i) {
            if (k + i >= nchunks) break;
            const float alpha = expf(c[i]);
            p[tile_of(k + i) * pn4] = st;
            st.x = alpha * st.x + u[i].x;
            st.y = alpha * st.y + u[i].y;
            st.z = alpha * st.z + u[i].z;
            st.w = alpha * st.w + u[i].w;
        }
#pragma unroll
        for (int i = 0; i < kWalkTiles; ++i) {
            u[i] = un[i];
            c[i] = cn[i];
        }
    }
    if (end != nullptr && inside) reinterpret_cast<float4*>(end)[edge] = st;
}

template <bool REVERSE>
int launch_state_walk(const SsdShape& s, float* states, const float* cs, const float* start, float* end,
                      cudaStream_t stream) {
    if (!aligned16(states, start, end)) return SSD_ERR_ALIGN;
    const int n4 = state_cols(s) / 4;
    const size_t total = static_cast<size_t>(s.batch) * s.nheads * kStateRows * n4;
    const size_t blocks = (total + kWalkThreads - 1) / kWalkThreads;
    if (blocks > 0x7fffffff) return SSD_ERR_RANGE;
    launch_plain(state_walk_kernel<REVERSE>, static_cast<unsigned>(blocks), kWalkThreads, 0, stream, states, cs, start,
                 end, s.seqlen / kTile, n4, s.seqlen, s.headdim, s.dstate / 4, total);
    return launch_status();
}

// ------------------------------------------------------------------ read-only fold of the recurrence
// acc <- exp(cs_last,k) * acc + terms[k], walked over the tiles forward (reverse = 0: the state after the
// last tile from the per-tile contributions U_k) or backward (reverse = 1: the gradient of the state before
// the first tile from the local dS_k).  Nothing is written but the [P,N] result: the sequence-parallel
// mode uses it to learn a rank's outflow before it knows its inflow.
__global__ void __launch_bounds__(256)
state_fold_kernel(const float* __restrict__ terms, const float* __restrict__ cs, const float* __restrict__ start,
                  float* __restrict__ result, int nchunks, int pn4, int seqlen, size_t total, int reverse) {
    after_previous();
    allow_next();
    const size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const size_t bh = idx / pn4;
    const int e = static_cast<int>(idx % pn4);
    const float4* p = reinterpret_cast<const float4*>(terms) + bh * nchunks * pn4 + e;
    const float* csl = cs + bh * seqlen + (kTile - 1);
    float4 acc = start ? reinterpret_cast<const float4*>(start)[bh * pn4 + e] : make_float4(0.f, 0.f, 0.f, 0.f);
    auto tile_of = [&](int i) { return reverse ? nchunks - 1 - i : i; };
    float4 u = p[static_cast<size_t>(tile_of(0)) * pn4];
    for (int i = 0; i < nchunks; ++i) {
        const float4 cur = u;
        if (i + 1 < nchunks) u = p[static_cast<size_t>(tile_of(i + 1)) * pn4];
        const float alpha = expf(csl[static_cast<size_t>(tile_of(i)) * kTile]);
        acc.x = alpha * acc.x + cur.x;
        acc.y = alpha * acc.y + cur.y;
        acc.z = alpha * acc.z + cur.z;
        acc.w = alpha * acc.w + cur.w;
    }
    reinterpret_cast<float4*>(result)[bh * pn4 + e] = acc;
}

// ------------------------------------------------------------------ backward state passing with g_last
// CTA = one (b,h); thread owns ELEMS float4 of the [P,N] state.  dstates holds
// the local dS_k on entry and dU_k (gradient reaching chunk k's own state
// contribution, i.e. d loss / d S_{k+1}) on exit.  g_last[b,h,k] =
// alpha_k * sum(dU_k * S_k) is the gradient w.r.t. cs_last of chunk k.
// The block reduction is a fixed tree, so results are run-to-run identical.
constexpr int kPartTiles = 384;  // tiles whose per-warp partials share the 48 KB of shared memory
template <int ELEMS, bool LONG>
__global__ void __launch_bounds__(1024)
state_passing_bwd_kernel(float* __restrict__ dstates, const float* __restrict__ states_start,
                         const float* __restrict__ cs, const float* __restrict__ dfinal, float* __restrict__ g_last,
                         float* __restrict__ d_initial, int nchunks, int seqlen) {
    after_previous();
    allow_next();
    extern __shared__ float part[];  // [min(nchunks, kPartTiles)][32]: per-warp partial dot products
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const size_t bh = blockIdx.x;
    const int pn4 = ELEMS * 1024;
    float4* dp = reinterpret_cast<float4*>(dstates) + bh * nchunks * pn4;
    const float4* sp = reinterpret_cast<const float4*>(states_start) + bh * nchunks * pn4;
    const float* csl = cs + bh * seqlen + (kTile - 1);
    float4 g[ELEMS], ds_n[ELEMS], st_n[ELEMS];
#pragma unroll
    for (int i = 0; i < ELEMS; ++i) {
        g[i] = dfinal ? reinterpret_cast<const float4*>(dfinal)[bh * pn4 + i * 1024 + tid] : make_float4(0, 0, 0, 0);
        const size_t o = static_cast<size_t>(nchunks - 1) * pn4 + i * 1024 + tid;
        ds_n[i] = dp[o];
        st_n[i] = sp[o];
    }
    if constexpr (!LONG) {
        // No block-wide barrier inside the walk over the tiles: each warp reduces its own products and
        // parks the partial; the loads of the next tile are always in flight before this tile's stores.
        for (int k = nchunks - 1; k >= 0; --k) {
            const float alpha = expf(csl[static_cast<size_t>(k) * kTile]);
            float dot = 0.f;
#pragma unroll
            for (int i = 0; i < ELEMS; ++i) {
                const size_t o = static_cast<size_t>(k) * pn4 + i * 1024 + tid;
                const float4 ds = ds_n[i];
                const float4 st = st_n[i];
                if (k > 0) {
                    ds_n[i] = dp[o - pn4];
                    st_n[i] = sp[o - pn4];
                }
                dp[o] = g[i];
                dot += g[i].x * st.x + g[i].y * st.y + g[i].z * st.z + g[i].w * st.w;
                g[i].x = ds.x + alpha * g[i].x;
                g[i].y = ds.y + alpha * g[i].y;
                g[i].z = ds.z + alpha * g[i].z;
                g[i].w = ds.w + alpha * g[i].w;
            }
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, d);
            if (lane == 0) part[k * 32 + warp] = dot;
        }
        __syncthreads();
        for (int k = warp; k < nchunks; k += 32) {
            float v = part[k * 32 + lane];
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
            if (lane == 0) g_last[bh * nchunks + k] = expf(csl[static_cast<size_t>(k) * kTile]) * v;
        }
    } else {
        // More tiles than partials fit the shared memory (sequences beyond 49152 tokens): the same walk in
        // blocks of kPartTiles tiles, with the fixed-order reduction of a block's partials between two blocks.
        for (int k_hi = nchunks; k_hi > 0; k_hi -= kPartTiles) {
            const int k_lo = k_hi > kPartTiles ? k_hi - kPartTiles : 0;
            for (int k = k_hi - 1; k >= k_lo; --k) {
                const float alpha = expf(csl[static_cast<size_t>(k) * kTile]);
                float dot = 0.f;
#pragma unroll
                for (int i = 0; i < ELEMS; ++i) {
                    const size_t o = static_cast<size_t>(k) * pn4 + i * 1024 + tid;
                    const float4 ds = ds_n[i];
                    const float4 st = st_n[i];
                    if (k > 0) {
                        ds_n[i] = dp[o - pn4];
                        st_n[i] = sp[o - pn4];
                    }
                    dp[o] = g[i];
                    dot += g[i].x * st.x + g[i].y * st.y + g[i].z * st.z + g[i].w * st.w;
                    g[i].x = ds.x + alpha * g[i].x;
                    g[i].y = ds.y + alpha * g[i].y;
                    g[i].z = ds.z + alpha * g[i].z;
                    g[i].w = ds.w + alpha * g[i].w;
                }
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, d);
                if (lane == 0) part[(k - k_lo) * 32 + warp] = dot;
            }
            __syncthreads();
            for (int k = k_lo + warp; k < k_hi; k += 32) {
                float v = part[(k - k_lo) * 32 + lane];
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
                if (lane == 0) g_last[bh * nchunks + k] = expf(csl[static_cast<size_t>(k) * kTile]) * v;
            }
            if (k_lo > 0) __syncthreads();  // the partials are read before the next block overwrites them
        }
    }
    if (d_initial != nullptr) {
#pragma unroll
        for (int i = 0; i < ELEMS; ++i) reinterpret_cast<float4*>(d_initial)[bh * pn4 + i * 1024 + tid] = g[i];
    }
}

// ------------------------------------------------------------------ ddt transpose, dA and d(dt_bias)
// One launch, two kinds of CTA.  The first batch * tiles * ceil(H / 32) CTAs turn ddt_t [B,H,L] into ddt [B,L,H], a
// [128 tokens x up to 32 heads] patch each through shared memory.  The last H CTAs reduce one head each, in fp64 and
// in a fixed order: dA[h] over the per-tile partials, d(dt_bias)[h] (if asked for) over the head's rows of ddt_t.  A head
// that the kernels treat as `parts` heads has that many rows and partials, which are added up here.
__device__ __forceinline__ double block_sum_256(double v, double* red, int tid) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    __syncthreads();
    if ((tid & 31) == 0) red[tid >> 5] = v;
    __syncthreads();
    return ((red[0] + red[1]) + (red[2] + red[3])) + ((red[4] + red[5]) + (red[6] + red[7]));
}

// ALIGNED: ddt_t, the caller's buffer, takes 16-byte loads.
template <bool ALIGNED>
__device__ __forceinline__ float4 load_quad(const float* p) {
    if constexpr (ALIGNED) return *reinterpret_cast<const float4*>(p);
    return make_float4(p[0], p[1], p[2], p[3]);
}

template <bool ALIGNED>
__global__ void __launch_bounds__(256)
dt_finalize_kernel(const float* __restrict__ ddt_t, const double* __restrict__ part, float* __restrict__ ddt,
                   float* __restrict__ dA, float* __restrict__ ddt_bias, int batch, int nchunks, int nheads, int parts,
                   int tokens, int head_blocks, int head_bits) {
    after_previous();
    allow_next();
    __shared__ float patch[kTile][33];
    __shared__ double red[8];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int turns = batch * nchunks * head_blocks;
    const int seqlen = nchunks * kTile;
    if (static_cast<int>(blockIdx.x) < turns) {
        const int k = blockIdx.x % nchunks, rest = blockIdx.x / nchunks;
        const int h0 = rest % head_blocks * 32, b = rest / head_blocks;
        const int heads = min(32, nheads - h0);
        float4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (warp + 8 * i < heads) {
                const float* src = ddt_t + (static_cast<size_t>(b) * nheads + h0 + warp + 8 * i) * parts * seqlen + k * kTile + 4 * lane;
                v[i] = load_quad<ALIGNED>(src);
                for (int j = 1; j < parts; ++j) {
                    const float4 o = load_quad<ALIGNED>(src + static_cast<size_t>(j) * seqlen);
                    v[i].x += o.x;
                    v[i].y += o.y;
                    v[i].z += o.z;
                    v[i].w += o.w;
                }
            }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (warp + 8 * i >= heads) break;
            patch[4 * lane][warp + 8 * i] = v[i].x;
            patch[4 * lane + 1][warp + 8 * i] = v[i].y;
            patch[4 * lane + 2][warp + 8 * i] = v[i].z;
            patch[4 * lane + 3][warp + 8 * i] = v[i].w;
        }
        __syncthreads();
        const int hh = tid & ((1 << head_bits) - 1);
        if (hh >= heads) return;
        float* dst = ddt + (static_cast<size_t>(b) * tokens + k * kTile) * nheads + h0 + hh;
        const int t_end = min(kTile, tokens - k * kTile);
        for (int t = tid >> head_bits; t < t_end; t += 256 >> head_bits) dst[static_cast<size_t>(t) * nheads] = patch[t][hh];
        return;
    }
    const int h = blockIdx.x - turns;
    double acc = 0.0;
    const int per_head = parts * nchunks;  // the parts of a head are neighbours
    for (int i = tid; i < batch * per_head; i += 256) {
        const int b = i / per_head, k = i - b * per_head;
        acc += part[(static_cast<size_t>(b) * nheads + h) * per_head + k];
    }
    acc = block_sum_256(acc, red, tid);
    if (tid == 0) dA[h] = static_cast<float>(acc);
    if (ddt_bias == nullptr) return;
    acc = 0.0;
    for (int b = 0; b < batch; ++b) {
        const float* row = ddt_t + (static_cast<size_t>(b) * nheads + h) * parts * seqlen;
#pragma unroll 4
        for (int i = tid; i < parts * (seqlen / 4); i += 256) {
            const float4 f = load_quad<ALIGNED>(row + 4 * static_cast<size_t>(i));
            acc += (static_cast<double>(f.x) + f.y) + (static_cast<double>(f.z) + f.w);
        }
    }
    acc = block_sum_256(acc, red, tid);
    if (tid == 0) ddt_bias[h] = static_cast<float>(acc);
}

// log2 of the smallest power of two that holds the heads of a block (at most 32)
int head_bits_of(int nheads) {
    int bits = 0;
    while (bits < 5 && (1 << bits) < nheads) ++bits;
    return bits;
}

}  // namespace

}  // namespace ssd

extern "C" int ssd_dt_cumsum(const SsdShape* shape, const float* dt, const float* dt_bias, const float* A, float* q,
                             float* cs, ssd_stream_t stream) {
    using namespace ssd;
    const int rc = ssd_check_shape(shape);
    if (rc != SSD_OK) return rc;
    if (!dt || !A || !q || !cs) return SSD_ERR_NULL;
    const dim3 grid(shape->seqlen / kTile, (shape->nheads + 31) / 32, shape->batch);
    launch_plain(dt_cumsum_kernel, grid, 256, 0, reinterpret_cast<cudaStream_t>(stream), dt, dt_bias, A, q, cs, *shape,
                 head_bits_of(shape->nheads));
    return launch_status();
}

extern "C" int ssd_state_passing_fwd(const SsdShape* shape, float* states, const float* cs,
                                     const float* initial_state, float* final_state, ssd_stream_t stream) {
    using namespace ssd;
    const int rc = ssd_check_shape(shape);
    if (rc != SSD_OK) return rc;
    if (!states || !cs) return SSD_ERR_NULL;
    return launch_state_walk<false>(*shape, states, cs, initial_state, final_state, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int ssd_state_fold(const SsdShape* shape, const float* terms, const float* cs, const float* start,
                              float* result, int reverse, ssd_stream_t stream) {
    using namespace ssd;
    const int rc = ssd_check_shape(shape);
    if (rc != SSD_OK) return rc;
    if (!terms || !cs || !result) return SSD_ERR_NULL;
    if (has_extents(*shape)) return SSD_ERR_UNSUPPORTED;
    const int pn4 = shape->headdim * shape->dstate / 4;
    const size_t total = static_cast<size_t>(shape->batch) * shape->nheads * pn4;
    const unsigned blocks = static_cast<unsigned>((total + 255) / 256);
    launch_plain(state_fold_kernel, blocks, 256, 0, reinterpret_cast<cudaStream_t>(stream), terms, cs, start, result,
                 shape->seqlen / kTile, pn4, shape->seqlen, total, reverse != 0);
    return launch_status();
}

extern "C" int ssd_state_passing_bwd(const SsdShape* shape, float* dstates, const float* states_start, const float* cs,
                                     const float* dfinal, float* g_last, float* d_initial, ssd_stream_t stream) {
    using namespace ssd;
    const int rc = ssd_check_shape(shape);
    if (rc != SSD_OK) return rc;
    if (!dstates || !cs || (g_last && !states_start)) return SSD_ERR_NULL;
    if (g_last && has_extents(*shape)) return SSD_ERR_UNSUPPORTED;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (!g_last) return launch_state_walk<true>(*shape, dstates, cs, dfinal, d_initial, st);
    const unsigned blocks = static_cast<unsigned>(shape->batch) * shape->nheads;
    const int nchunks = shape->seqlen / kTile;
    const size_t part_bytes = static_cast<size_t>(nchunks < kPartTiles ? nchunks : kPartTiles) * 32 * sizeof(float);
    const bool lng = nchunks > kPartTiles;
    auto launch = [&](auto kernel) {
        launch_plain(kernel, blocks, 1024, part_bytes, st, dstates, states_start, cs, dfinal, g_last, d_initial,
                     nchunks, shape->seqlen);
    };
    if (shape->dstate == 64) {
        lng ? launch(state_passing_bwd_kernel<1, true>) : launch(state_passing_bwd_kernel<1, false>);
    } else {
        lng ? launch(state_passing_bwd_kernel<2, true>) : launch(state_passing_bwd_kernel<2, false>);
    }
    return launch_status();
}

extern "C" int ssd_dt_finalize_bias_bwd(const SsdShape* shape, const float* ddt_t, const double* dA_partial, float* ddt,
                                        float* dA, float* ddt_bias, ssd_stream_t stream) {
    using namespace ssd;
    const int rc = ssd_check_shape(shape);
    if (rc != SSD_OK) return rc;
    if (!ddt_t || !dA_partial || !ddt || !dA) return SSD_ERR_NULL;
    const int parts = head_parts(*shape), heads = shape->nheads / parts;
    const int nchunks = shape->seqlen / kTile, head_blocks = (heads + 31) / 32;
    const int64_t blocks = static_cast<int64_t>(shape->batch) * nchunks * head_blocks + heads;
    if (blocks > 0x7fffffff) return SSD_ERR_RANGE;
    launch_plain(aligned16(ddt_t) ? dt_finalize_kernel<true> : dt_finalize_kernel<false>, static_cast<unsigned>(blocks), 256, 0, reinterpret_cast<cudaStream_t>(stream),
                 ddt_t, dA_partial, ddt, dA, ddt_bias, shape->batch, nchunks, heads, parts, row_tokens(*shape),
                 head_blocks, head_bits_of(heads));
    return launch_status();
}

extern "C" int ssd_dt_finalize_bwd(const SsdShape* shape, const float* ddt_t, const double* dA_partial, float* ddt,
                                   float* dA, ssd_stream_t stream) {
    return ssd_dt_finalize_bias_bwd(shape, ddt_t, dA_partial, ddt, dA, nullptr, stream);
}
