// Backward of the feature transformer as a dense product of whole numbers on the tensor pipe, for tables of few rows.
//
// The table gradient of a row block is  one_hot^T [rows x pairs]  times  gradients [pairs x columns].  The walk over row lists
// (ft_backward_tiled_kernel) adds 32 floats per clock and SM out of shared memory; the tensor pipe does 8192 multiply-adds of
// bytes, zeros included.  With 27 of 147 rows active in every pair (ataxx) the dense product needs 44 times the walk's
// operations in eight digits at 256 times its rate, and no row lists.  Time of the backward with 147 rows and 32768 positions,
// walk / product: 256 columns 83 / 41 us, 1024 columns 323 / 134 (b200_net::bwd_mma draws the line between the two).
//
// Numbers.  A gradient times a power of two, chosen so that the largest there can be (`gmax`) stays below 2^22, is a sum of eight
// signed bytes down to units of 2^-37 (take_piece): eight rows of the product's first factor.  All 24 bits of a gradient down to
// 2^-36 of the largest there can be are in these; what smaller ones have below the last digit is added to their rows by fp32
// atomics.  Sums of bytes are exact in the 32-bit accumulators (for kUnitStepsMost steps of 128 pairs), so that a sum is rounded to
// fp32 only when its eight digits are put together (four times) and when its parts of several CTAs are added.  (Four digits in
// units of 2^-31 of the largest, 33 us at 256 columns, left columns of small output weights and positions of small errors fewer
// bits than fp32 does: over seven decades of weights and six of errors single sums were off by up to 2e-2 of their magnitudes.)  A gmax that is not finite takes a slow path of fp32 atomics:
// infinities and NaN reach the rows they belong to and no others.
//
// ft_onehot_kernel (a CTA per chunk of at most 128 pairs, once per batch) writes the one-hot factor as bits.  In
// ft_backward_mma_kernel a CTA holds the sums of all rows x 32 columns x eight digits in tensor memory.  Three groups of four
// warps, each with a stage of shared memory of its own, write the digits and the one-hot bytes of every third step; one thread
// issues the products; its warpgroup takes finished sums out, puts the digits together and adds them to the gradient.
#pragma once
#include "bulk_copy.cuh"
#include "kernels_ft.cuh"

namespace b200 {

constexpr int kStepPairs = 128;  // pairs per step (and chunk): a row of 128 bytes in both factors
constexpr int kMmaStages = 3, kMmaGroupThreads = 128;
constexpr int kMmaThreads = (1 + kMmaStages) * kMmaGroupThreads;
constexpr int kUnitCols = 32;  // gradient columns of a unit: with four digits the 128 lanes of tensor memory, so that eight take two tiles
constexpr int kDigitBytes = 128 * kStepPairs;  // of a tile
constexpr int kUnitStepsMost = 256;  // sums of digits stay below 2^22, where a pair holds a row 64 times below 2^28
constexpr int kMmaTileRows = 256;    // most rows of the one-hot tile: three stages fit into shared memory, both tiles' sums into tensor memory
constexpr int kUnitFixed = 4;        // what taking out a unit's sums costs, in steps

// Rows of the one-hot tile: the table's, one that all pairs hold (its sums are the bias gradient), and up to whole loads of sums.
__host__ __device__ inline int ft_mma_rows(int R) { return (R + 1 + 31) & ~31; }
// One-hot bits of a chunk: of each of 128 threads, the 16 pairs 16 (thread % 8) .. + 15 of the rows thread / 8 + 16 q, eight q in 16
// bytes, the threads' pieces side by side.
__host__ __device__ inline int ft_mma_words(int rows) { return (rows + 127) / 128; }  // 16-byte pieces per thread
__host__ __device__ inline int ft_mma_ent_cap(int R) { return ft_mma_words(ft_mma_rows(R)) * kMmaGroupThreads * 8; }
constexpr int kStepHead = 4 + kStepPairs;  // ints per chunk: whether a pair holds a row twice, three unused, the pair ids (-1: none)
__host__ __device__ inline size_t ft_mma_smem(int rows) { return 1024 + (size_t)kMmaStages * (2 * kDigitBytes + rows * kStepPairs); }

// Byte of (row, k) in a tile of 128-byte rows with the 128-byte swizzle.
__device__ __forceinline__ uint32_t swizzled(uint32_t row, uint32_t k) { return row * 128 + (((k >> 4) ^ (row & 7)) << 4) + (k & 15); }

// Latency bound, one load deep; beside the step before unless the batch is a network's first.
constexpr int kOnehotThreads = 1024;
static __global__ void __launch_bounds__(kOnehotThreads) ft_onehot_kernel(TileArgs t) {
    __shared__ uint32_t seen[kMmaTileRows * 4];  // a bit per (row, pair)
    __shared__ int twice;
    const int4 chunk = t.chunks[blockIdx.x];
    if (chunk.z == 0) return;  // (the launch is sized from the batch size alone)
    const int c0 = chunk.y, cn = chunk.z, Q = t.list_len / 8;
    static_assert(kOnehotThreads >= kStepPairs * 8, "a thread per eight slots: one load's latency");
    const int pair = threadIdx.x / Q, q = threadIdx.x - pair * Q;
    int len = 0, id = -1;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (pair < cn) {
        len = __ldg(&t.pairs[c0 + pair].y) - 8 * q;
        v = __ldg(reinterpret_cast<const uint4*>(t.lists + (size_t)(c0 + pair) * t.list_len) + q);
    }
    if ((int)threadIdx.x < cn) id = __ldg(&t.pairs[c0 + threadIdx.x].x);
    for (int k = threadIdx.x; k < kMmaTileRows * 4; k += kOnehotThreads) seen[k] = 0;
    if (threadIdx.x == 0) twice = 0;
    __syncthreads();
    const uint32_t w[4] = {v.x, v.y, v.z, v.w}, bit = 1u << (pair & 31);
#pragma unroll
    for (int h = 0; h < 8; h++)
        if (h < len && (atomicOr(&seen[(h & 1 ? w[h >> 1] >> 16 : w[h >> 1] & 0xffffu) * 4 + (pair >> 5)], bit) & bit)) twice = 1;
    if (threadIdx.x < 4) {
        const int held = min(32, max(0, cn - 32 * (int)threadIdx.x));
        seen[t.block_rows * 4 + threadIdx.x] = held == 32 ? ~0u : (1u << held) - 1u;
    }
    __syncthreads();
    int* head = t.csr_start + (size_t)blockIdx.x * t.start_cap;
    if (threadIdx.x == 0) *reinterpret_cast<int4*>(head) = make_int4(twice, 0, 0, 0);
    if (threadIdx.x < kStepPairs) head[4 + threadIdx.x] = id;
    uint32_t* out = reinterpret_cast<uint32_t*>(t.csr_ent + (size_t)blockIdx.x * t.ent_cap);
    for (int k = threadIdx.x; k < t.ent_cap / 2; k += kOnehotThreads) {  // sixteen pairs of two rows a word
        const int owner = k / 4 % kMmaGroupThreads, row = owner / 8 + 16 * (k / (4 * kMmaGroupThreads) * 8 + k % 4 * 2), c = owner % 8;
        auto pairs16 = [&](int row) { return row < kMmaTileRows ? seen[row * 4 + c / 2] >> 16 * (c & 1) & 0xffffu : 0u; };
        out[k] = pairs16(row) | pairs16(row + 16) << 16;
    }
}

// ---- tensor memory and the products

// Descriptors of the factors' tiles by their low words (the high ones are alike): the address / 16, so that 32 bytes on is 2 more.
constexpr uint32_t kTileHigh = 64u | 1u << 14 | 2u << 29;  // eight rows are 1024 bytes, 128-byte swizzle
__device__ __forceinline__ uint32_t tile_low(uint32_t smem) { return (smem & 0x3ffffu) >> 4 | 1u << 16; }
__device__ __forceinline__ uint32_t byte_product(int n) {  // signed bytes, 32-bit sums, M = 128
    return 2u << 4 | 1u << 7 | 1u << 10 | (uint32_t)(n >> 3) << 17 | 8u << 24;
}
__device__ __forceinline__ void multiply_bytes(uint32_t sums, uint32_t a, uint32_t b, uint32_t form, bool add) {
    asm volatile(
        "{\n.reg .pred p;\n.reg .b64 da, db;\nmov.b64 da, {%1, %5};\nmov.b64 db, {%2, %5};\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], da, db, %3, p;\n}" ::"r"(sums),
        "r"(a), "r"(b), "r"(form), "r"((int)add), "r"(kTileHigh)
        : "memory");
}
__device__ __forceinline__ void products_done(uint64_t* bar) {  // arrives when all products issued so far are finished
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void sums_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void sums_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void load_sums16(uint32_t at, int (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
          "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(at)
        : "memory");
}
// what has been loaded is there (the words pass through, so that nothing reads them before)
__device__ __forceinline__ void loaded_sums(int (&v)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]), "+r"(v[9]), "+r"(v[10]),
                   "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15])::"memory");
}
__device__ __forceinline__ bool mbar_try_wait_long(uint64_t* bar, uint32_t parity) {  // asleep for some us
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 4000;\nselp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// ---- the division of the work
// The line of units: block by block, inside a block by units of 32 columns, inside these step by step; a unit weighs its steps and
// kUnitFixed more.  A CTA takes a piece of the line.
struct MmaPlace {
    int block, unit, step, before;  // before: steps of the line that come before this one
};
// The first step at or after weight `cut` of the line.  A whole warp.
__device__ __forceinline__ MmaPlace ft_mma_place(const TileArgs& t, int units, long long cut, int lane) {
    long long base = 0, steps = 0;
    for (int b0 = t.first_block; b0 < t.last_block; b0 += 32) {
        const int b = b0 + lane;
        const int n = b < t.last_block ? t.chunk_begin[b + 1] - t.chunk_begin[b] : 0;
        const int w = n ? n + kUnitFixed : 0;
        int w_incl = w, n_incl = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int wu = __shfl_up_sync(0xffffffffu, w_incl, o), nu = __shfl_up_sync(0xffffffffu, n_incl, o);
            if (lane >= o) w_incl += wu, n_incl += nu;
        }
        const long long first = base + (long long)units * (w_incl - w);
        const bool here = n > 0 && cut >= first && cut < first + (long long)units * w;
        MmaPlace p{};
        if (here) {
            const int r = (int)(cut - first);
            p.block = b;
            p.unit = r / w;
            p.step = min(r - p.unit * w, n);
            p.before = (int)(steps + (long long)units * (n_incl - n)) + p.unit * n + p.step;
        }
        const unsigned m = __ballot_sync(0xffffffffu, here);
        if (m) {
            const int from = __ffs(m) - 1;
            p.block = __shfl_sync(0xffffffffu, p.block, from);
            p.unit = __shfl_sync(0xffffffffu, p.unit, from);
            p.step = __shfl_sync(0xffffffffu, p.step, from);
            p.before = __shfl_sync(0xffffffffu, p.before, from);
            return p;
        }
        base += (long long)units * __shfl_sync(0xffffffffu, w_incl, 31);
        steps += (long long)units * __shfl_sync(0xffffffffu, n_incl, 31);
    }
    return {t.last_block, 0, 0, (int)steps};
}
__device__ __forceinline__ long long ft_mma_line(const TileArgs& t, int units, int lane) {
    long long line = 0;
    for (int b0 = t.first_block; b0 < t.last_block; b0 += 32) {
        const int b = b0 + lane, n = b < t.last_block ? t.chunk_begin[b + 1] - t.chunk_begin[b] : 0;
        line += __reduce_add_sync(0xffffffffu, n ? n + kUnitFixed : 0);
    }
    return line * units;
}
// A walk along the steps of a piece.
struct MmaWalk {
    int block, unit, step, left, steps, chunk0;  // of the step it stands on; `left`: steps of the piece from here on
    __device__ __forceinline__ void enter(const TileArgs& t) {  // the step may lie just past its unit
        if (left <= 0) return;
        chunk0 = __ldg(t.chunk_begin + block);
        steps = __ldg(t.chunk_begin + block + 1) - chunk0;
    }
    __device__ __forceinline__ void settle(const TileArgs& t, int units) {
        while (left > 0 && step >= steps) {
            step -= steps;
            if (++unit < units) continue;
            unit = 0;
            do {
                block++;
                enter(t);
            } while (steps == 0);
        }
    }
    __device__ __forceinline__ void advance(const TileArgs& t, int units, int by) {
        left -= by;
        step += by;
        settle(t, units);
    }
    __device__ __forceinline__ int chunk() const { return chunk0 + step; }
    // steps from here on until the sums are taken out
    __device__ __forceinline__ int run() const { return min(left, min(steps - step, kUnitStepsMost - step % kUnitStepsMost)); }
};

// One gradient in fp32 for the slow path (column `col` of the pair's H pre-activations).
template <bool PAIRWISE, bool ONE>
__device__ __forceinline__ float ft_gradient_at(const FtArgs& a, int pair, int col) {
    const int width = PAIRWISE ? a.H / 2 : a.H, c = PAIRWISE && col >= width ? col - width : col;
    const float d = ONE ? a.w1[((size_t)2 * a.out_bucket[pair >> 1] + (pair & 1)) * width + c] * a.dout[pair >> 1] : a.dx[(size_t)pair * width + c];
    if (!PAIRWISE) return d * ft_act_bwd(a.act, a.x[(size_t)pair * a.H + col]);
    const float* u = a.u + (size_t)pair * a.H;
    return (d * u[col < width ? col + width : c]) * ft_act_bwd(1, u[col]);
}
// v where 0 < y < 1, else 0: for outputs of the clamp (bits of positive floats order as the floats do)
__device__ __forceinline__ float inside_only(float y, float v) { return __float_as_uint(y) - 1u < 0x3f7fffffu ? v : 0.f; }

// Its value times a power of two, of the products' operands: d is dx (or w1 x dout) times that power, y the activation output of the
// column, for pairwise networks y and other those of the two sides.
template <bool PAIRWISE, bool ONE, bool SQUARE>
__device__ __forceinline__ float ft_scaled_gradient(float d, float y, float other, int side) {
    if (PAIRWISE) return side ? inside_only(other, __fmul_rn(d, y)) : inside_only(y, __fmul_rn(d, other));
    return SQUARE ? __fmul_rn(d, ft_act_bwd(ONE ? 3 : 2, y)) : inside_only(y, d);
}

// The digits of a scaled gradient, |v| < 2^22 - 2^15, from whole multiples of 1, 2^-22 and 2^-37: the sum with 1.5 x 2^23 of these is
// rounded to one, which its low bits hold.  Returned: three, three and two low bytes of a digit each, with 0x80 added to the first
// two (by 0x8080 more of the multiples) and 0x40 to the third; v becomes the rest.
__device__ __forceinline__ uint32_t take_piece(float& v, int piece) {
    const float shift = (12582912.f + 32896.f) / (piece == 0 ? 1.f : piece == 1 ? 4194304.f : 137438953472.f);
    const float sum = __fadd_rn(v, shift);  // (never one operation with the product that v is)
    v = __fsub_rn(v, __fsub_rn(sum, shift));
    return __float_as_uint(sum);
}
// What the i-th digit counts.
__device__ __forceinline__ float digit_weight(int i) {
    const int bits = i < 3 ? 8 * i : i < 6 ? 8 * (i - 3) - 22 : 8 * (i - 6) - 37;
    return __uint_as_float((uint32_t)(127 + bits) << 23);
}

// grid = one CTA per SM.  All waits are for the CTA's own warps and products, and bounded.
// Bound by the groups' instructions and the latency between them: a step (128 pairs x 32 columns, 160 rows) takes 2150 clocks, its
// products 640 of them; half of the issue slots are taken.  The operands of a group's next step are loaded as soon as those of this
// one have become digits: 41 us at 256 columns instead of 46 with the loads behind the step.  (Lists of the set bytes in shared
// memory, to set and to clear them, instead of writing the whole tile from bits, in the form of four digits: 52 instead of 40 us.  In
// more parts than one, for blocks of 768 rows, the digits are made once for each, and it loses to the walk: 420 against 282 us at
// 16384 x 2048, where the 64-byte pieces of a pairwise row cost as much again.)
template <bool PAIRWISE, bool ONE, bool SQUARE>
__global__ void __launch_bounds__(kMmaThreads, 1) ft_backward_mma_kernel(FtArgs a, TileArgs t) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full[kMmaStages], empty[kMmaStages], done, taken, last;
    __shared__ uint32_t sums_at;
    __shared__ MmaPlace piece[2];
    __shared__ int dead_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rows = ft_mma_rows(t.block_rows), width = PAIRWISE ? a.H / 2 : a.H;
    constexpr int kCols = PAIRWISE ? kUnitCols / 2 : kUnitCols;  // columns of x of a unit
    const int units = (width + kCols - 1) / kCols;
    unsigned char* base = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    const int stage_bytes = 2 * kDigitBytes + rows * kStepPairs;
    volatile int* dead = &dead_s;
    if (tid == 0) {
        for (int s = 0; s < kMmaStages; s++) mbar_init(&full[s], kMmaGroupThreads), mbar_init(&empty[s], 1);
        mbar_init(&done, 1), mbar_init(&taken, 128), mbar_init(&last, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        dead_s = 0;
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&sums_at)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (warp == 0) {  // (the batch's tables are older than the step)
        const long long line = ft_mma_line(t, units, lane);
        const MmaPlace p0 = ft_mma_place(t, units, line * blockIdx.x / gridDim.x, lane), p1 = ft_mma_place(t, units, line * (blockIdx.x + 1) / gridDim.x, lane);
        if (lane == 0) piece[0] = p0, piece[1] = p1;
    }
    step_begin(a.stamp);
    sums_fence_before();
    __syncthreads();
    sums_fence_after();
    const uint32_t sums = sums_at;
    // Scaled by 2^k, no gradient is above 2^22 - 2^15.
    const unsigned m0 = __ldcg(a.gmax), m1 = ONE ? __ldcg(a.gmax + 1) : 0u;
    const float bound = __uint_as_float(m0) * (ONE ? __uint_as_float(m1) : 1.f) * (SQUARE ? 2.f : 1.f) * 1.015625f;
    const bool finite = m0 < 0x7f800000u && m1 < 0x7f800000u && bound < __uint_as_float(0x7f800000u);
    const int k = min(120, 148 - (int)(__float_as_uint(bound) >> 23));
    const float scale = __uint_as_float((uint32_t)(127 + k) << 23), unit = __uint_as_float((uint32_t)(127 - k) << 23);

    MmaWalk walk{piece[0].block, piece[0].unit, piece[0].step, finite && bound > 0.f ? piece[1].before - piece[0].before : 0, 0, 0};
    walk.enter(t);
    walk.settle(t, units);
    auto wait = [&](uint64_t* bar, uint32_t parity) {
        for (int tries = 0; tries < 1000000; tries++)
            if (mbar_try_wait_long(bar, parity) || *dead) return;
        *dead = 1;  // everybody runs on to the end without waiting; the host hears of it
        *a.gave_up = 1;
    };

    if (!finite) {
        for (int ch = t.chunk_begin[t.first_block] + (int)blockIdx.x; ch < t.chunk_begin[t.last_block]; ch += gridDim.x) {
            const int4 chunk = t.chunks[ch];
            for (int i = warp; i < chunk.z; i += kMmaThreads / 32) {
                const int2 pair = t.pairs[chunk.y + i];
                const uint16_t* list = t.lists + (size_t)(chunk.y + i) * t.list_len;
                for (int col = lane; col < a.H; col += 32) {
                    const float g = ft_gradient_at<PAIRWISE, ONE>(a, pair.x, col);
                    if (g == 0.f) continue;
                    atomicAdd(a.g_bias + col, g);
                    for (int e = 0; e < pair.y; e++) atomicAdd(a.g_table + ((size_t)chunk.x * t.block_rows + list[e]) * a.H + col, g);
                }
            }
        }
    } else if (warp < 4) {  // products (a thread of warp 0) and, when a unit's are finished, its sums out, each warp those of its 32 lanes
        asm volatile("setmaxnreg.dec.sync.aligned.u32 104;");
        const int d = lane >> 3, at = ((lane & 7) - 2 * warp) & 7;
        const int c = 8 * warp + 4 * (at & 1) + (at >> 1);  // this lane's gradient column in the unit
        const float by_high = digit_weight(d), by_low = digit_weight(4 + d);
        const uint32_t form = byte_product(rows), step16 = stage_bytes >> 4;
        const uint32_t digits0 = tile_low(smem_u32(base)), hot0 = tile_low(smem_u32(base + 2 * kDigitBytes));
        int stage = 0, unit_no = 0;
        uint32_t phase = 0;
        for (int n; walk.left > 0; walk.advance(t, units, n), unit_no++) {
            n = walk.run();
            if (warp == 0) {
                if (lane == 0) {
                    if (unit_no > 0) wait(&taken, (unit_no - 1) & 1);
                    sums_fence_after();
                    for (int s = 0; s < n; s++) {
                        const uint32_t digits = digits0 + stage * step16, hot = hot0 + stage * step16;
                        wait(&full[stage], phase);
                        sums_fence_after();
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            multiply_bytes(sums, digits + 2 * q, hot + 2 * q, form, s > 0 || q > 0);
                            multiply_bytes(sums + kMmaTileRows, digits + kDigitBytes / 16 + 2 * q, hot + 2 * q, form, s > 0 || q > 0);
                        }
                        products_done(&empty[stage]);
                        if (++stage == kMmaStages) stage = 0, phase ^= 1;
                    }
                    products_done(&done);
                }
                __syncwarp();
            }
            const int x_col = walk.unit * kCols + (PAIRWISE ? c & 15 : c), col = PAIRWISE && c >= 16 ? width + x_col : x_col;
            float* to = a.g_table + ((size_t)walk.block * t.block_rows + d) * a.H + col;
            const int own_rows = x_col < width ? t.block_rows - d : -1;
            float* bias = a.g_bias + col;
            wait(&done, unit_no & 1);
            __syncwarp();
            sums_fence_after();
            const size_t four = (size_t)4 * a.H;
            for (int n0 = 0; n0 < rows; n0 += 16) {
                int high[16], low[16];
                load_sums16(sums + n0 + ((uint32_t)warp << 21), high);
                load_sums16(sums + kMmaTileRows + n0 + ((uint32_t)warp << 21), low);
                loaded_sums(high);
                loaded_sums(low);
                float sum[4];
#pragma unroll
                for (int g = 0; g < 4; g++) {
                    // four rows of the table, two digits of eight: a lane ends up with all of row d's
                    float f[4];
#pragma unroll
                    for (int r = 0; r < 4; r++) f[r] = fmaf((float)low[4 * g + r], by_low, (float)high[4 * g + r] * by_high);
                    const float a2 = (d & 1 ? f[1] : f[0]) + __shfl_xor_sync(0xffffffffu, d & 1 ? f[0] : f[1], 8);
                    const float b2 = (d & 1 ? f[3] : f[2]) + __shfl_xor_sync(0xffffffffu, d & 1 ? f[2] : f[3], 8);
                    sum[g] = ((d & 2 ? b2 : a2) + __shfl_xor_sync(0xffffffffu, d & 2 ? a2 : b2, 16)) * unit;
                }
#pragma unroll
                for (int g = 0; g < 4; g++)
                    if (n0 + 4 * g == own_rows && sum[g] != 0.f) atomicAdd(bias, sum[g]);
                // (added also where nobody else adds: a caller that clears the gradients itself may have several passes summed)
#pragma unroll
                for (int g = 0; g < 4; g++, to += four)
                    if (n0 + 4 * g < own_rows && sum[g] != 0.f) atomicAdd(to, sum[g]);
            }
            sums_fence_before();
            mbar_arrive(&taken);
        }
        if (warp == 0 && lane == 0) {
            products_done(&last);  // nothing is in flight when the CTA ends
            for (int tries = 0; tries < 1000000 && !mbar_try_wait_long(&last, 0); tries++) {}
        }
        __syncwarp();
    } else {  // digits and one-hot bytes
        asm volatile("setmaxnreg.inc.sync.aligned.u32 136;");
        const int group = (warp >> 2) - 1, w4 = warp & 3, tg = w4 * 32 + lane;  // of steps group, group + 3, ...
        unsigned char* digits = base + group * stage_bytes;
        unsigned char* hot = digits + 2 * kDigitBytes;
        // this lane's four columns (m) and its pairs: T sets of four
        constexpr int T = PAIRWISE ? 1 : 2;
        const int m = PAIRWISE ? lane & 3 : lane & 7;
        const int quad = PAIRWISE ? lane >> 2 & 3 : lane >> 3;  // which four of sixteen pairs
        auto sixteen = [&](int e) { return PAIRWISE ? w4 + 4 * (lane >> 4) : w4 + 4 * e; };
        float4 y0[T][4], y1[PAIRWISE ? T : 1][4], dd[ONE ? 1 : T][4];
        float dout[ONE ? T : 1][4];
        int w1_row[ONE ? T : 1][4];
        int4 ids[T];
        constexpr int kWords = kMmaTileRows / 128;
        const int words16 = ft_mma_words(rows);
        uint4 bits[kWords];
        int cu = 0, chunk = 0;  // unit of columns and chunk of the step in the making
        auto fetch_ids = [&]() {  // of the step that `walk` stands on
            if (walk.left > 0)
#pragma unroll
                for (int e = 0; e < T; e++) ids[e] = __ldg(reinterpret_cast<const int4*>(t.csr_start + (size_t)walk.chunk() * t.start_cap + 4) + 4 * sixteen(e) + quad);
        };
        // and, these being there, the operands of a part, when those of the step before have been used
        auto fetch = [&](int part) {
            if (walk.left <= 0 || (PAIRWISE && part == 0)) return;
            const int e = PAIRWISE ? 0 : part, col = min(walk.unit * kCols + 4 * m, width - 4);
#pragma unroll
            for (int p = 0; p < 4; p++) {
                const int id = p == 0 ? ids[e].x : p == 1 ? ids[e].y : p == 2 ? ids[e].z : ids[e].w, pair = max(id, 0);  // (of a pair that is none, no byte is set)
                const float* y = (PAIRWISE ? a.u : a.x) + (size_t)pair * a.H + col;
                y0[e][p] = ld_once4(reinterpret_cast<const float4*>(y));
                if (PAIRWISE) y1[e][p] = ld_once4(reinterpret_cast<const float4*>(y + width));
                if (ONE) {
                    dout[e][p] = __ldcg(a.dout + (pair >> 1));
                    w1_row[e][p] = 2 * __ldg(a.out_bucket + (pair >> 1)) + (pair & 1);
                } else {
                    dd[e][p] = ld_fresh4(reinterpret_cast<const float4*>(a.dx + (size_t)pair * width + col));
                }
            }
        };
        int twice = 0;
        auto fetch_bits = [&]() {
            if (walk.left <= 0) return;
            twice = __ldg(t.csr_start + (size_t)walk.chunk() * t.start_cap);
            const uint4* src = reinterpret_cast<const uint4*>(t.csr_ent + (size_t)walk.chunk() * t.ent_cap) + tg;
#pragma unroll
            for (int q = 0; q < kWords; q++)
                if (q < words16) bits[q] = __ldg(src + q * kMmaGroupThreads);
        };
        // The digits are made and stored in two parts (sets of pairs, PAIRWISE: sides), the first while the stage is still in use.
        uint32_t words[4][8];  // [column][digit] of four pairs each
        uint32_t below = 0;    // whether any gradient of a part has bits below the last digit
        auto make = [&](int part) {
            const int e = PAIRWISE ? 0 : part;
            below = 0;
            if (ONE && (!PAIRWISE || part == 0)) {  // (the unit's weights are a few KB, in L1)
                const int col = min(cu * kCols + 4 * m, width - 4);
#pragma unroll
                for (int p = 0; p < 4; p++) dd[0][p] = scale4(__ldg(reinterpret_cast<const float4*>(a.w1 + (size_t)w1_row[e][p] * width + col)), dout[e][p]);
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                uint32_t q[3][4];
#pragma unroll
                for (int p = 0; p < 4; p++) {
                    auto comp = [&](const float4& v) { return j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w; };
                    float rest = ft_scaled_gradient<PAIRWISE, ONE, SQUARE>(__fmul_rn(comp(dd[ONE ? 0 : e][p]), scale), comp(y0[e][p]), PAIRWISE ? comp(y1[e][p]) : 0.f, part);
#pragma unroll
                    for (int piece = 0; piece < 3; piece++) q[piece][p] = take_piece(rest, piece);
                    below |= __float_as_uint(rest) & 0x7fffffffu;
                }
                // four pairs' digit of this column: one word
                uint32_t* to = words[j];
#pragma unroll
                for (int piece = 0; piece < 3; piece++) {
                    const uint32_t a01 = __byte_perm(q[piece][0], q[piece][1], 0x5140), a23 = __byte_perm(q[piece][2], q[piece][3], 0x5140);
                    to[3 * piece] = __byte_perm(a01, a23, 0x5410) ^ 0x80808080u;
                    to[3 * piece + 1] = __byte_perm(a01, a23, 0x7632) ^ 0x80808080u;
                    if (piece < 2)
                        to[3 * piece + 2] = (__byte_perm(__byte_perm(q[piece][0], q[piece][1], 0x0062), __byte_perm(q[piece][2], q[piece][3], 0x0062), 0x5410) + 0x40404040u) ^ 0x80808080u;
                }
            }
        };
        // What the digits leave of a part's gradients, by atomics: of gradients below 2^-36 of the largest there can be.
        auto add_rest = [&](int part) {
            const int4 c = __ldg(t.chunks + chunk);
            for (int i = 0; i < 16; i++) {
                const int in_chunk = 16 * sixteen(PAIRWISE ? 0 : part) + 4 * quad + (i & 3), x_col = cu * kCols + 4 * m + (i >> 2);
                if (in_chunk >= c.z || x_col >= width) continue;
                const int2 pair = __ldg(t.pairs + c.y + in_chunk);
                const float* y = (PAIRWISE ? a.u : a.x) + (size_t)pair.x * a.H + x_col;
                const float dx = ONE ? __fmul_rn(a.w1[((size_t)2 * a.out_bucket[pair.x >> 1] + (pair.x & 1)) * width + x_col], a.dout[pair.x >> 1]) : a.dx[(size_t)pair.x * width + x_col];
                float rest = ft_scaled_gradient<PAIRWISE, ONE, SQUARE>(__fmul_rn(dx, scale), y[0], PAIRWISE ? y[width] : 0.f, part);
                for (int piece = 0; piece < 3; piece++) take_piece(rest, piece);
                if (rest == 0.f) continue;
                const int col = PAIRWISE && part ? width + x_col : x_col;
                atomicAdd(a.g_bias + col, rest * unit);
                const uint16_t* list = t.lists + (size_t)(c.y + in_chunk) * t.list_len;
                for (int k = 0; k < pair.y; k++) atomicAdd(a.g_table + ((size_t)c.x * t.block_rows + __ldg(list + k)) * a.H + col, rest * unit);
            }
        };
        auto store_words = [&](int part) {
            const int e = PAIRWISE ? 0 : part, side = PAIRWISE ? part : 0;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const uint32_t mm = m + 4 * side, s8 = (mm + 2 * j) & 7;
                uint32_t* to = reinterpret_cast<uint32_t*>(digits + ((mm >> 1) * 32 + s8) * 128 + ((sixteen(e) ^ s8) << 4) + 4 * quad);
#pragma unroll
                for (int d = 0; d < 8; d++) to[(d >> 2) * (kDigitBytes / 4) + 256 * (d & 3)] = words[j][d];
            }
        };
        unsigned char* own_hot = hot + (tg >> 3) * 128 + (((tg & 7) ^ (tg >> 3 & 7)) << 4);  // 16 pairs of rows tg / 8 + 16 q
        auto store_bits = [&]() {
#pragma unroll
            for (int q = 0; q < kWords * 8; q++) {
                if (16 * q >= rows) break;
                const uint4 v = bits[q / 8];
                const uint32_t pick = q % 8 / 2, word = pick == 0 ? v.x : pick == 1 ? v.y : pick == 2 ? v.z : v.w, b = q & 1 ? word >> 16 : word;
                *reinterpret_cast<uint4*>(own_hot + q * 2048) =
                    make_uint4((b & 15u) * 0x00204081u & 0x01010101u, (b >> 4 & 15u) * 0x00204081u & 0x01010101u, (b >> 8 & 15u) * 0x00204081u & 0x01010101u,
                               (b >> 12 & 15u) * 0x00204081u & 0x01010101u);
            }
        };
        // a pair holds a row more than once: the bytes are counts, from the prepared lists
        auto store_counts = [&]() {
#pragma unroll
            for (int q = 0; q < kWords; q++) bits[q] = make_uint4(0, 0, 0, 0);
            store_bits();
            asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(kMmaGroupThreads) : "memory");
            const int4 c = __ldg(t.chunks + chunk);
            if (tg < c.z) {
                hot[swizzled(t.block_rows, tg)] = 1;
                const uint16_t* list = t.lists + (size_t)(c.y + tg) * t.list_len;
                for (int e = 0, len = __ldg(&t.pairs[c.y + tg].y); e < len; e++) {
                    const uint32_t byte = swizzled(__ldg(list + e), tg);
                    atomicAdd(reinterpret_cast<unsigned*>(hot + (byte & ~3u)), 1u << 8 * (byte & 3u));
                }
            }
        };
        walk.advance(t, units, group);
        fetch_ids();
        fetch(0);
        fetch(1);
        fetch_bits();
        for (uint32_t phase = 1; walk.left > 0; phase ^= 1) {
            cu = walk.unit;
            chunk = walk.chunk();
            walk.advance(t, units, kMmaStages);
            fetch_ids();
            make(0);
            wait(&empty[group], phase);  // (the first round finds the stage free)
            __syncwarp();
            store_words(0);
            fetch(0);
            if (below) add_rest(0);
            make(1);
            store_words(1);
            fetch(1);
            if (below) add_rest(1);
            if (twice) store_counts();
            else store_bits();
            fence_proxy_async();
            mbar_arrive(&full[group]);
            fetch_bits();
        }
    }
    __syncthreads();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(sums));
}

}  // namespace b200
