// y[M,N] = x[M,K] * w[N,K]^T (+ residual) for the projections of a Mamba-2 block, fp32 in and out, on tcgen05.
//
// fp32 products on the CUDA cores are what bounds these projections (two library calls of 131 and 59 us per block at
// 16384 tokens, 75% of the network's forward).  Each operand is split into THREE bf16 parts (hi + mid + lo: all 24 bits of
// an fp32 significand) and the six products of weight 2^-16 and above are formed,
//
//     hi*lo + mid*mid + lo*hi   (2^-16)      hi*mid + mid*hi   (2^-8)      hi*hi
//
// The tensor core truncates where it adds to its fp32 accumulator, which is a bias on sums of one sign and grows with the
// number of additions of full size.  So an accumulator holds 64 columns of K only, smallest products first: four additions
// of full size.  It is then added to the running sum in registers, rounded to nearest.
//
// One CTA = 128 rows x a run of 96-column tiles.  x goes to tensor memory once (three parts of up to 192 columns of K: 288
// columns; two 96-column accumulators take 192 of the rest, so that one is read out under the other's products); w arrives by
// TMA from its split copy, one tile of all parts per stage, two stages.  K beyond 192 is taken in equal chunks of up
// to 192 (the last one filled up with zeros by the loads), with the sums of two tiles kept in registers.  The issue of the products
// bounds a tile (72 of them at K = 192, 3.5 us); before the first, a chunk of x is loaded (the later ones under the products of the
// chunk before) and converted.
//
// [16384,192] x [902,192]: 43 us with the split of w, 50 from cold caches (139 in the library); [16384,384] x [192,384] + residual:
// 29, 36 (66 without the residual).  One accumulator for all of K: 45 and 27 us.  Error against 64
// bits, relative 2-norm, operands of both signs / of one sign (the library's fp32 kernel in brackets): K = 192 8.6e-8 / 9.2e-8
// (2.5e-7 / 2.1e-7), K = 384 9.2e-8 / 9.4e-8 (3.5e-7 / 2.9e-7), K = 1536 1.2e-7 / 1.1e-7 (7.0e-7 / 5.8e-7).  With one accumulator
// for all of K it was 1.8e-7 / 2.7e-7, 3.5e-7 / 6.1e-7 and 1.5e-6 / 3.7e-6.  Measured and dropped: 64-column tiles in three
// stages, CTAs starting at different tiles.
#include "ssd_host.h"
#include "ssd_pdl.cuh"
#include "ssd_tile.cuh"

namespace ssd {

namespace {

constexpr int kLinCols = 96;                              // columns of a tile
constexpr int kLinMaxBlocks = 3;                          // 64-column blocks of K per chunk
constexpr uint32_t kLinBox = kLinCols * 128;              // one part of one block: [96 x 64] bf16
constexpr int kLinWarps = 8;                              // convert x, add up and write the result (two warps per 32 rows)
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

// v = hi + mid + lo, bf16 each.  An infinity becomes (+-1, 0, +-inf): its lo part meets only the other operand's hi part,
// which has that operand's sign and is zero with it, so the sum is the infinity or NaN that fp32 gives (an infinity minus itself
// would be NaN, and an infinite hi part would meet mid and lo parts of either sign).
__device__ __forceinline__ void split3(float v, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    const uint32_t sign = __float_as_uint(v) >> 16 & 0x8000u, magnitude = __float_as_uint(v) & 0x7FFFFFFFu;
    if (magnitude >= 0x7F800000u) {
        hi = magnitude == 0x7F800000u ? sign | 0x3F80u : 0x7FC0u;
        mid = 0;
        lo = magnitude == 0x7F800000u ? sign | 0x7F80u : 0u;
        return;
    }
    hi = magnitude >= 0x7F7F8000u ? sign | 0x7F7Fu : pack_bf16x2(v, 0.f) & 0xFFFFu;  // the largest bf16 instead of an infinity
    const float rest = v - __uint_as_float(hi << 16);
    mid = pack_bf16x2(rest, 0.f) & 0xFFFFu;
    lo = pack_bf16x2(rest - __uint_as_float(mid << 16), 0.f) & 0xFFFFu;
}
__device__ __forceinline__ void split3_pair(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    hi = pack_bf16x2(a, b);
    if ((hi & 0x7F80u) == 0x7F80u || (hi & 0x7F800000u) == 0x7F800000u) {
        uint32_t h, m, l;
        split3(a, hi, mid, lo);
        split3(b, h, m, l);
        hi |= h << 16;
        mid |= m << 16;
        lo |= l << 16;
        return;
    }
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
// HELD: tiles whose sums a CTA keeps at once; 2 with several chunks of K, which are the outer loop (a CTA then has no more tiles).
template <int BLOCKS, int HELD>
__global__ void __launch_bounds__(kLinThreads, 1)
linear_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const LinearArgs a,
              int* status) {
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr int blocks = BLOCKS;
    constexpr uint32_t stage_bytes = lin_stage_bytes(blocks);
    float* patches = reinterpret_cast<float*>(smem + 2 * stage_bytes);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 2 * stage_bytes + kLinWarps * kLinPatch);
    uint64_t* full_x = bars;          // a chunk of x has landed
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
    // Stage of a tile of w in the pass over a chunk of K, and the stage where that chunk of x lands on its way to tensor
    // memory: the one of the pass before's first tile, so that it arrives under that pass's second.
    auto stage_of = [](int pass, int t) { return (pass + t) & 1; };
    auto x_stage = [&](int pass) { return stage_of(pass, 1); };

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
            mbar_init(&acc_free[i], kLinWarps);
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
            int sum = 0;          // accumulators so far
            uint32_t parity = 0;  // of full_w, a bit per stage
            for (int pass = 0; pass < a.chunks; ++pass) {
                mbar_wait(x_ready, pass & 1, status, kStatusMmaTimeout | wait_site(7, 1));
                for (int t = 0; t < ntiles; ++t) {
                    const int st = stage_of(pass, t);
                    mbar_wait(&full_w[st], (parity >> st) & 1u, status, kStatusMmaTimeout | wait_site(7, 2));
                    parity ^= 1u << st;
                    const uint32_t base = smem_u32(smem) + st * stage_bytes;
#pragma unroll
                    for (int blk = 0; blk < blocks; ++blk, ++sum) {
                        if (sum >= 2)  // what it held before has been read
                            mbar_wait(&acc_free[sum & 1], ((sum >> 1) - 1) & 1, status, kStatusMmaTimeout | wait_site(7, 3));
                        tc_fence_after_sync();
                        const uint32_t acc = tmem + (sum & 1) * kLinCols;
                        uint32_t accumulate = 0u;
                        auto product = [&](int xp, int wp) {
                            const uint64_t w0 = operand_desc0(base + wp * blocks * kLinBox, kLinBox, false);
#pragma unroll
                            for (int s = 4 * blk; s < 4 * blk + 4; ++s) {
                                umma_bf16_ta(acc, tm_x + xp * part_cols + 8u * s, w0 + (kstep_offset(kLinBox, false, s) >> 4), idesc,
                                             accumulate);
                                accumulate = 1u;
                            }
                        };
                        product(0, 2);
                        product(1, 1);
                        product(2, 0);
                        product(0, 1);
                        product(1, 0);
                        product(0, 0);
                        umma_commit(&acc_ready[sum & 1]);
                    }
                    umma_commit(&done[st]);
                }
            }
        }
    } else if (warp == kLinWarps + 1) {  // ---- issues the loads
        if (lane == 0) {
            uint32_t busy = 0, parity = 0;      // stages that products read, and the parity of done, a bit per stage
            auto stage_idle = [&](int st) {     // the products of the tile it holds are done
                if (((busy >> st) & 1u) == 0) return;
                mbar_wait(&done[st], (parity >> st) & 1u, status, kStatusMmaTimeout | wait_site(7, 4));
                parity ^= 1u << st;
                busy ^= 1u << st;
            };
            for (int pass = 0; pass < a.chunks; ++pass) {
                const int k0 = pass * blocks * 64;
                auto load_w = [&](int t) {
                    const int st = stage_of(pass, t);
                    stage_idle(st);
                    busy |= 1u << st;
                    mbar_arrive_expect_tx(&full_w[st], stage_bytes);
                    for (int part = 0; part < 3; ++part)
                        for (int blk = 0; blk < blocks; ++blk)  // 64 bf16 columns seen as 32 floats
                            tma_load_2d(smem + st * stage_bytes + (part * blocks + blk) * kLinBox, &map_w, &full_w[st],
                                        (k0 + blk * 64) / 2, part * a.cols_padded + (tile0 + t) * kLinCols);
                };
                stage_idle(x_stage(pass));
                mbar_arrive_expect_tx(full_x, 2u * blocks * kSlabBytes);
                for (int i = 0; i < 2 * blocks; ++i)
                    tma_load_2d(smem + x_stage(pass) * stage_bytes + i * kSlabBytes, &map_x, full_x, k0 + 32 * i, row0);
                load_w(0);
                mbar_wait(x_ready, pass & 1, status, kStatusMmaTimeout | wait_site(7, 5));  // x has left its stage
                for (int t = 1; t < ntiles; ++t) load_w(t);
            }
        }
    } else {  // ---- convert x, write the result
        const int quarter = warp & 3, half = warp >> 2;  // 32 rows; every other slab of x, half the columns of a tile
        constexpr int kCols = kLinCols / 2;
        const int out_row = row0 + quarter * 32;
        float* patch = patches + warp * 32 * (kLinPatchCols + 1);
        float sums[HELD][kCols];  // this thread's row
        auto clear = [&]() {
#pragma unroll
            for (int i = 0; i < HELD * kCols; ++i) sums[i / kCols][i % kCols] = 0.f;
        };
        if constexpr (HELD > 1) clear();
        int sum = 0;  // accumulators so far
        auto add_up = [&](float* total) {
            const int acc = sum & 1;
            ok = mbar_wait(&acc_ready[acc], (sum >> 1) & 1, status, kStatusMmaTimeout | wait_site(7, 7)) && ok;
            tc_fence_after_sync();
            float v[kCols];
#pragma unroll
            for (int c = 0; c < kCols; c += 16) tmem_ld16(tmem_addr(tmem + acc * kLinCols, warp, half * kCols + c), v + c);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < kCols; ++i) total[i] += v[i];
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_free[acc]);
            ++sum;
        };
        auto write_tile = [&](const float* total, int t) {  // eight columns at a time, turned so that a row is contiguous
            const int col = (tile0 + t) * kLinCols + half * kCols + (lane & 7), r0 = lane >> 3;
            const size_t o = static_cast<size_t>(out_row + r0) * a.cols + col;
            // of this thread's rows r0, r0 + 4, ... those that exist
            const int rows = ok ? static_cast<int>(max(0ll, min(8ll, (a.rows - out_row - r0 + 3) / 4))) : 0;
            auto inside = [&](int c0, int i) { return i < rows && col + c0 < a.cols; };
            constexpr int kPatches = kCols / kLinPatchCols, kAtOnce = HELD == 1 ? kPatches : 3;  // residual loads in flight together
#pragma unroll
            for (int j0 = 0; j0 < kPatches; j0 += kAtOnce) {
                float add[kAtOnce][8];
#pragma unroll
                for (int j = 0; j < kAtOnce; ++j)
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int c0 = (j0 + j) * kLinPatchCols;
                        add[j][i] = a.residual != nullptr && inside(c0, i) ? a.residual[o + c0 + static_cast<size_t>(4 * i) * a.cols] : 0.f;
                    }
#pragma unroll
                for (int j = 0; j < kAtOnce; ++j) {
                    const int c0 = (j0 + j) * kLinPatchCols;
#pragma unroll
                    for (int i = 0; i < kLinPatchCols; ++i) patch[lane * (kLinPatchCols + 1) + i] = total[c0 + i];
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        if (inside(c0, i))
                            a.out[o + c0 + static_cast<size_t>(4 * i) * a.cols] =
                                patch[(r0 + 4 * i) * (kLinPatchCols + 1) + (lane & 7)] + add[j][i];
                    __syncwarp();
                }
            }
        };
        for (int pass = 0; pass < a.chunks; ++pass) {
            // every accumulator of the pass before has been read: its products are done and x's tensor memory may be replaced
            ok = mbar_wait(full_x, pass & 1, status, kStatusTmaTimeout | wait_site(7, 6)) && ok;
            tc_fence_after_sync();
#pragma unroll 1
            for (int slab = half; slab < 2 * blocks; slab += 2) {
                const uint8_t* src = smem + x_stage(pass) * stage_bytes + slab * kSlabBytes;
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
            if constexpr (HELD == 1) {
                for (int t = 0; t < ntiles; ++t) {
                    clear();
#pragma unroll
                    for (int blk = 0; blk < blocks; ++blk) add_up(sums[0]);
                    write_tile(sums[0], t);
                }
            } else {
#pragma unroll
                for (int t = 0; t < HELD; ++t)
                    if (t < ntiles) {
#pragma unroll
                        for (int blk = 0; blk < blocks; ++blk) add_up(sums[t]);
                        if (pass == a.chunks - 1) write_tile(sums[t], t);  // under the next tile's products
                    }
            }
        }
    }
    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 512);
}

// Chunks of K and blocks of 64 columns in a chunk: as few as hold all of K, as even as they come; 0 if K is not made of blocks.
int linear_chunks(int k) { return k <= 0 || k % 64 != 0 ? 0 : (k / 64 + kLinMaxBlocks - 1) / kLinMaxBlocks; }
int linear_blocks(int k) {
    const int chunks = linear_chunks(k);
    return chunks == 0 ? 0 : (k / 64 + chunks - 1) / chunks;
}
int linear_cols_padded(int cols) { return (cols + kLinCols - 1) / kLinCols * kLinCols; }

}  // namespace

}  // namespace ssd

// The kernel's own latency for one round of CTAs is 13 to 17 us with one chunk of K and 10 us more with each further one; below
// these sizes the library's fp32 kernel takes less.  Measured over K = 64 ... 1536, 64 to 6278 columns, 200 to 16384 rows (us, this
// kernel / the library): [1024,192] x [902,192] 17 / 17, [2048,192] x [902,192] 22 / 26, [16384,192] x [902,192] 50 / 139;
// [2048,384] x [902,384] 34 / 41, [4096,384] x [192,384] 32 / 25; [2048,576] x [576,576] 44 / 33, [512,576] x [2438,576] 44 / 50;
// [16384,1024] x [192,1024] 81 / 150.  Fewer columns than a tile's 96 were slower at every size (64 columns: 16384 rows, K = 192
// 20 / 18, 30000 rows, K = 768 81 / 76).  Of the sizes taken none was slower.
extern "C" int ssd_linear_pays(long long rows, int cols, int k) {
    const int chunks = ssd::linear_chunks(k);
    if (rows <= 0 || cols <= 0 || chunks == 0) return 0;
    return cols >= ssd::kLinCols && static_cast<double>(rows) * cols * k >= 2.3e8 * chunks ? 1 : 0;
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
    a.chunks = linear_chunks(k);
    a.tiles = a.cols_padded / kLinCols;
    const int sms = sm_count();
    if (sms <= 0) return SSD_ERR_LAUNCH;
    const int64_t row_tiles = (rows + 127) / 128;
    // with several chunks a CTA keeps its sums over all of them: at most two tiles; otherwise few row tiles are given
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
    auto launch = [&](auto kernel, std::atomic<uint64_t>& smem_set) {
        const int r = set_max_smem_once(reinterpret_cast<const void*>(kernel), lin_smem_bytes(blocks), smem_set);
        if (r != SSD_OK) return r;
        launch_tiles(row_tiles * items, kernel, dim3(static_cast<unsigned>(row_tiles), items), kLinThreads, lin_smem_bytes(blocks),
                     st, map_x, map_w, a, status);
        return launch_status();
    };
    static std::atomic<uint64_t> smem_set[5];
    if (a.chunks > 1)  // 256 columns of K or more: chunks of two or three blocks
        return blocks == 3 ? launch(linear_kernel<3, 2>, smem_set[0]) : launch(linear_kernel<2, 2>, smem_set[1]);
    return blocks == 3   ? launch(linear_kernel<3, 1>, smem_set[2])
           : blocks == 2 ? launch(linear_kernel<2, 1>, smem_set[3])
                         : launch(linear_kernel<1, 1>, smem_set[4]);
}
