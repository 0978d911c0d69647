// y[M,N] = x[M,K] * w[N,K]^T (+ residual) for the projections of a Mamba-2 block, fp32 in and out, on tcgen05.
//
// fp32 products on the CUDA cores are what bounds these projections (two library calls of 131 and 59 us per block at
// 16384 tokens, 75% of the network's forward).  Each operand is split into THREE bf16 parts (hi + mid + lo: all 24 bits of
// an fp32 significand) and the six products of weight 2^-16 and above are formed,
//
//     hi*lo + mid*mid + lo*hi   (2^-16)      hi*mid + mid*hi   (2^-8)      hi*hi
//
// smallest first, because the tensor core truncates where it adds to the fp32 accumulator: only the K/16 hi*hi additions
// meet a sum of full size.  Error against 64 bits, normal operands, relative 2-norm: K = 192 1.6e-7 (the library's fp32
// kernel: 2.5e-7), K = 384 3.2e-7 (3.5e-7).
//
// One CTA = 128 rows x a run of 96-column tiles.  x goes to tensor memory once (three parts of up to 192 columns of K: 288
// columns; two 96-column accumulators take 192 of the rest, so a tile is written out under the next one's
// products); w arrives by TMA from its split copy, one tile of all parts per stage, two stages.  K beyond 192 is
// taken in chunks: first the small products of every chunk, then hi*hi of every chunk, so that the order above holds for
// the whole sum; the chunks of x but the last are converted twice.  The issue of the products bounds a tile (72 of them at K =
// 192, 3.5 us); before the first, a pass loads and converts its chunk of x (3 to 5 us).
// [16384,192] x [902,192]: 41 us (132 in the library); [16384,384] x [192,384] + residual: 25 us (65).  Measured and dropped:
// 64-column tiles in three stages (46 and 30 us), CTAs starting at different tiles (no change).
#include "ssd_host.h"
#include "ssd_pdl.cuh"
#include "ssd_tile.cuh"

namespace ssd {

namespace {

constexpr int kLinCols = 96;                              // columns of a tile
constexpr int kLinMaxBlocks = 3;                          // 64-column blocks of K per chunk
constexpr uint32_t kLinBox = kLinCols * 128;              // one part of one block: [96 x 64] bf16
constexpr int kLinWarps = 8;                              // convert x (two warps per 32 rows), write the result (four per tile)
constexpr int kLinThreads = kLinWarps * 32 + 64;          // and the issuing and the producer warp
constexpr int kLinPatchCols = 8;
constexpr uint32_t kLinPatch = 32 * (kLinPatchCols + 1) * sizeof(float);  // per warp: 32 rows x 8 columns on their way out

struct LinearArgs {
    const float* residual;
    float* out;
    long long rows;
    int cols, cols_padded, chunks, tiles, tiles_per_item;
};

__host__ __device__ constexpr uint32_t lin_stage_bytes(int blocks) { return 3u * blocks * kLinBox; }
__host__ __device__ constexpr uint32_t lin_smem_bytes(int blocks) {
    return 2 * lin_stage_bytes(blocks) + kLinWarps * kLinPatch + 256;
}
static_assert(lin_smem_bytes(kLinMaxBlocks) <= 232448, "projection kernel exceeds the shared memory of one SM");
static_assert(128 * 128 * 2 <= 3 * kLinBox, "a block of x lands in the stage of a block of w");

// v = hi + mid + lo, bf16 each, for finite v (up to the largest bf16, 3.39e38)
__device__ __forceinline__ void split3_pair(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    hi = pack_bf16x2(a, b);
    const float a1 = a - __uint_as_float(hi << 16), b1 = b - __uint_as_float(hi & 0xFFFF0000u);
    mid = pack_bf16x2(a1, b1);
    lo = pack_bf16x2(a1 - __uint_as_float(mid << 16), b1 - __uint_as_float(mid & 0xFFFF0000u));
}

// w [cols, k] -> parts [3][cols_padded][k] bf16 (rows beyond cols are zero); one thread per pair.
__global__ void __launch_bounds__(256)
linear_split_kernel(const float* __restrict__ w, uint32_t* __restrict__ parts, int cols, int cols_padded, int k) {
    after_previous();
    allow_next();
    const size_t pairs = static_cast<size_t>(cols_padded) * k / 2;
    const size_t i = static_cast<size_t>(blockIdx.x) * 256 + threadIdx.x;
    if (i >= pairs) return;
    uint32_t hi = 0, mid = 0, lo = 0;
    if (i < static_cast<size_t>(cols) * k / 2) split3_pair(w[2 * i], w[2 * i + 1], hi, mid, lo);
    parts[i] = hi;
    parts[pairs + i] = mid;
    parts[2 * pairs + i] = lo;
}

// BLOCKS: 64-column blocks of K per chunk, a compile-time number, so that the issuing thread pays one addition per product.
template <int BLOCKS>
__global__ void __launch_bounds__(kLinThreads, 1)
linear_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const LinearArgs a,
              int* status) {
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr int blocks = BLOCKS;
    constexpr uint32_t stage_bytes = lin_stage_bytes(blocks);
    float* patches = reinterpret_cast<float*>(smem + 2 * stage_bytes);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 2 * stage_bytes + kLinWarps * kLinPatch);
    uint64_t* full_x = bars;          // a chunk of x has landed (in stage 1, and every product before it is done)
    uint64_t* x_ready = bars + 1;     // it is in tensor memory (per warp)
    uint64_t* full_w = bars + 2;      // [2] a tile of w has landed
    uint64_t* done = bars + 4;        // [2] the products that read a stage are done
    uint64_t* acc_ready = bars + 6;   // [2] an accumulator is complete
    uint64_t* acc_free = bars + 8;    // [2] it has been read (per warp)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 10);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row0 = blockIdx.x * 128;
    const int tile0 = blockIdx.y * a.tiles_per_item;
    const int ntiles = min(a.tiles_per_item, a.tiles - tile0);
    const int passes = 2 * a.chunks - 1;
    // pass -> chunk, and which products it forms
    auto chunk_of = [&](int pass) { return pass < a.chunks ? pass : 2 * a.chunks - 2 - pass; };
    auto has_small = [&](int pass) { return pass < a.chunks; };
    auto has_main = [&](int pass) { return pass >= a.chunks - 1; };
    // tiles that go through a stage in one pass
    auto per_pass = [&](int st) { return (ntiles + 1 - st) >> 1; };

    if ((smem_u32(smem) & 1023u) != 0) {  // the swizzled tiles need the declared alignment
        if (tid == 0) atomicCAS(status, 0, kStatusSmemAlign);
        return;
    }
    if (tid == 0) {
        mbar_init(full_x, 1);
        mbar_init(x_ready, kLinWarps);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&full_w[i], 1);
            mbar_init(&done[i], 1);
            mbar_init(&acc_ready[i], 1);
            mbar_init(&acc_free[i], 4);
        }
        fence_mbar_init();
    }
    if (warp == 0) tmem_alloc(tmem_slot, 512);
    after_previous();
    if (tid == 0) tmem_slot[1] = static_cast<uint32_t>(*reinterpret_cast<volatile int*>(status));
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    allow_next();
    if (tmem_slot[1] != 0) {  // an earlier kernel gave up on a bounded wait: leave without doing work
        if (warp == 0) tmem_dealloc(tmem, 512);
        return;
    }
    constexpr uint32_t part_cols = 32u * blocks;  // of a part of x in tensor memory (two bf16 per column)
    const uint32_t tm_x = tmem + 2 * kLinCols;
    static_assert(2 * kLinCols + 3 * 32 * kLinMaxBlocks <= 512, "tensor memory columns");
    bool ok = true;

    if (warp == kLinWarps) {  // ---- issues the products
        if (lane == 0) {
            const uint32_t idesc = make_idesc_bf16(128, kLinCols, false, false);
            for (int pass = 0; pass < passes; ++pass) {
                mbar_wait(x_ready, pass & 1, status, kStatusMmaTimeout | wait_site(7, 1));
                for (int t = 0; t < ntiles; ++t) {
                    const int st = t & 1;
                    mbar_wait(&full_w[st], (pass * per_pass(st) + (t >> 1)) & 1, status, kStatusMmaTimeout | wait_site(7, 2));
                    if (pass == 0 && t >= 2)  // its previous tile has been read
                        mbar_wait(&acc_free[st], ((t >> 1) - 1) & 1, status, kStatusMmaTimeout | wait_site(7, 3));
                    tc_fence_after_sync();
                    const uint32_t acc = tmem + st * kLinCols;
                    const uint32_t base = smem_u32(smem) + st * stage_bytes;
                    uint32_t accumulate = pass > 0 ? 1u : 0u;
                    auto product = [&](int xp, int wp) {
                        const uint64_t w0 = operand_desc0(base + wp * blocks * kLinBox, kLinBox, false);
#pragma unroll
                        for (int s = 0; s < 4 * blocks; ++s) {
                            umma_bf16_ta(acc, tm_x + xp * part_cols + 8u * s, w0 + (kstep_offset(kLinBox, false, s) >> 4), idesc,
                                         accumulate);
                            accumulate = 1u;
                        }
                    };
                    if (has_small(pass)) {
                        product(0, 2);
                        product(1, 1);
                        product(2, 0);
                        product(0, 1);
                        product(1, 0);
                    }
                    if (has_main(pass)) product(0, 0);
                    umma_commit(&done[st]);
                    if (pass == passes - 1) umma_commit(&acc_ready[st]);
                }
            }
        }
    } else if (warp == kLinWarps + 1) {  // ---- issues the loads
        if (lane == 0) {
            auto stage_idle = [&](int st, int loads) {  // the products of the last of its `loads` tiles so far are done
                if (loads > 0) mbar_wait(&done[st], (loads - 1) & 1, status, kStatusMmaTimeout | wait_site(7, 4));
            };
            for (int pass = 0; pass < passes; ++pass) {
                const int k0 = chunk_of(pass) * blocks * 64;
                auto load_w = [&](int t) {
                    const int st = t & 1;
                    mbar_arrive_expect_tx(&full_w[st], stage_bytes);
                    for (int part = 0; part < 3; ++part)
                        for (int blk = 0; blk < blocks; ++blk)  // 64 bf16 columns seen as 32 floats
                            tma_load_2d(smem + st * stage_bytes + (part * blocks + blk) * kLinBox, &map_w, &full_w[st],
                                        (k0 + blk * 64) / 2, part * a.cols_padded + (tile0 + t) * kLinCols);
                };
                // both stages idle: every product of the passes before is done, x's tensor memory may be replaced too
                stage_idle(0, pass * per_pass(0));
                stage_idle(1, pass * per_pass(1));
                mbar_arrive_expect_tx(full_x, 2u * blocks * kSlabBytes);
                for (int i = 0; i < 2 * blocks; ++i)
                    tma_load_2d(smem + stage_bytes + i * kSlabBytes, &map_x, full_x, k0 + 32 * i, row0);
                load_w(0);
                mbar_wait(x_ready, pass & 1, status, kStatusMmaTimeout | wait_site(7, 5));  // stage 1 has been read
                for (int t = 1; t < ntiles; ++t) {
                    if (t >= 2) stage_idle(t & 1, pass * per_pass(t & 1) + (t >> 1));
                    load_w(t);
                }
            }
        }
    } else {  // ---- convert x, write the result
        const int quarter = warp & 3, half = warp >> 2;
        const int out_row = row0 + quarter * 32;
        float* patch = patches + warp * 32 * (kLinPatchCols + 1);
        for (int pass = 0; pass < passes; ++pass) {
            ok = mbar_wait(full_x, pass & 1, status, kStatusTmaTimeout | wait_site(7, 6)) && ok;
            tc_fence_after_sync();
#pragma unroll 1
            for (int slab = half; slab < 2 * blocks; slab += 2) {
                const uint8_t* src = smem + stage_bytes + slab * kSlabBytes;
                uint32_t hi[16], mid[16], lo[16];
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const float4 f = *reinterpret_cast<const float4*>(src + swz(quarter * 32 + lane, c));
                    split3_pair(f.x, f.y, hi[2 * c], mid[2 * c], lo[2 * c]);
                    split3_pair(f.z, f.w, hi[2 * c + 1], mid[2 * c + 1], lo[2 * c + 1]);
                }
                tmem_st16(tmem_addr(tm_x, warp, 16 * slab), hi);
                tmem_st16(tmem_addr(tm_x + part_cols, warp, 16 * slab), mid);
                tmem_st16(tmem_addr(tm_x + 2 * part_cols, warp, 16 * slab), lo);
            }
            tmem_st_wait();
            signal_issuer(x_ready, lane);
        }
        for (int t = half; t < ntiles; t += 2) {  // one accumulator each
            const int st = half;
            ok = mbar_wait(&acc_ready[st], (t >> 1) & 1, status, kStatusMmaTimeout | wait_site(7, 7)) && ok;
            tc_fence_after_sync();
#pragma unroll 1
            for (int c0 = 0; c0 < kLinCols; c0 += kLinPatchCols) {
                float v[kLinPatchCols], add[kLinPatchCols];
                const int col = (tile0 + t) * kLinCols + c0 + (lane & 7), r0 = lane >> 3;
                const size_t o = static_cast<size_t>(out_row + r0) * a.cols + col;
                const bool inside = col < a.cols && ok;
#pragma unroll
                for (int i = 0; i < 8; ++i)  // rows r0, r0 + 4, ...
                    add[i] = a.residual != nullptr && inside && out_row + r0 + 4 * i < a.rows
                                 ? a.residual[o + static_cast<size_t>(4 * i) * a.cols] : 0.f;
                tmem_ld8(tmem_addr(tmem + st * kLinCols, warp, c0), v);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < kLinPatchCols; ++i) patch[lane * (kLinPatchCols + 1) + i] = v[i];
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (inside && out_row + r0 + 4 * i < a.rows)
                        a.out[o + static_cast<size_t>(4 * i) * a.cols] =
                            patch[(r0 + 4 * i) * (kLinPatchCols + 1) + (lane & 7)] + add[i];
                __syncwarp();
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_free[st]);
        }
    }
    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 512);
}

// Blocks of 64 in a chunk of K: the largest that divides it, at most three; 0 if K is not made of them.
int linear_blocks(int k) {
    if (k <= 0 || k % 64 != 0) return 0;
    for (int b = kLinMaxBlocks; b > 1; --b)
        if (k / 64 % b == 0) return b;
    return 1;
}
int linear_cols_padded(int cols) { return (cols + kLinCols - 1) / kLinCols * kLinCols; }

}  // namespace

}  // namespace ssd

// Below these sizes the kernel's own latency (10 us for one tile, 22 us with two chunks of K) exceeds the library's time:
// [784,192] x [902,192] 12 / 13 us, [196,192] x [902,192] 11 / 6.5; [4096,384] x [192,384] 25 / 22.
extern "C" int ssd_linear_pays(long long rows, int cols, int k) {
    const int blocks = ssd::linear_blocks(k);
    if (rows <= 0 || cols <= 0 || blocks == 0) return 0;
    const double work = static_cast<double>(rows) * cols * k;
    return work >= (k == 64 * blocks ? 1.6e8 : 4e8) ? 1 : 0;
}

extern "C" size_t ssd_linear_work_bytes(int cols, int k) {
    if (cols <= 0 || ssd::linear_blocks(k) == 0) return 0;
    return size_t(3) * ssd::linear_cols_padded(cols) * k * 2;
}

extern "C" int ssd_linear_fwd(const float* x, const float* w, const float* residual, float* out, long long rows, int cols,
                              int k, void* work, int* status, ssd_stream_t stream) {
    using namespace ssd;
    if (!x || !w || !out || !work || !status) return SSD_ERR_NULL;
    if (rows <= 0 || cols <= 0 || k <= 0) return SSD_ERR_SHAPE;
    const int blocks = linear_blocks(k);
    LinearArgs a{residual, out, rows, cols, linear_cols_padded(cols), 0, 0, 0};
    if (blocks == 0) return SSD_ERR_UNSUPPORTED;
    if (rows > 0x7fffffffLL - 128 || 3ll * a.cols_padded > 0x7fffffffLL) return SSD_ERR_RANGE;
    if (!aligned16(x, static_cast<const float*>(work))) return SSD_ERR_ALIGN;
    a.chunks = k / (64 * blocks);
    a.tiles = a.cols_padded / kLinCols;
    const int sms = sm_count();
    if (sms <= 0) return SSD_ERR_LAUNCH;
    const int64_t row_tiles = (rows + 127) / 128;
    // a chunked sum keeps its accumulators over all passes: at most two tiles per CTA; otherwise few row tiles are given
    // more CTAs along the columns
    a.tiles_per_item = a.chunks > 1 ? 2 : a.tiles / choose_head_split(row_tiles, a.tiles, sms, 1, 3);
    const int items = (a.tiles + a.tiles_per_item - 1) / a.tiles_per_item;
    if (items > 65535) return SSD_ERR_RANGE;
    CUtensorMap map_x, map_w;
    int rc = make_tmap_f32_2d(&map_x, x, static_cast<uint64_t>(rows), static_cast<uint64_t>(k), 128);
    if (rc == SSD_OK)
        rc = make_tmap_f32_2d(&map_w, work, 3ull * a.cols_padded, static_cast<uint64_t>(k) / 2, kLinCols);
    if (rc != SSD_OK) return rc;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const size_t pairs = static_cast<size_t>(a.cols_padded) * k / 2;
    launch_plain(linear_split_kernel, static_cast<unsigned>((pairs + 255) / 256), 256, 0, st, w,
                 static_cast<uint32_t*>(work), cols, a.cols_padded, k);
    rc = launch_status();
    if (rc != SSD_OK) return rc;
    static std::atomic<uint64_t> smem_set[kLinMaxBlocks];
    auto launch = [&](auto kernel, int b) {
        const int r = set_max_smem_once(reinterpret_cast<const void*>(kernel), lin_smem_bytes(b), smem_set[b - 1]);
        if (r != SSD_OK) return r;
        launch_tiles(row_tiles * items, kernel, dim3(static_cast<unsigned>(row_tiles), items), kLinThreads, lin_smem_bytes(b), st,
                       map_x, map_w, a, status);
        return launch_status();
    };
    return blocks == 3 ? launch(linear_kernel<3>, 3) : blocks == 2 ? launch(linear_kernel<2>, 2) : launch(linear_kernel<1>, 1);
}
