// The first dense layer of multi-layer networks (four or more rows per output bucket) on the tensor pipe: forward, gradient at
// its input, weight gradient.
//
// Semantics as in kernels_dense.cuh.  All three are streams over x or dx (K1 floats per position) with a contraction that is
// only M1 wide, so HBM bounds them: 8 KB per position and pass at K1 = 2048.  fp32 multiply-adds could not keep up with it
// (they held the kernels at a third of the copy rate); mma.sync does at a few per cent of its own rate, straight from
// registers, without the staging through shared memory and tensor memory that tcgen05 would add for a 16-wide product.
//
// An fp32 operand is split into three bf16 parts, each rounded to nearest: v = h + m + l exactly (8 bits each, short of
// numbers whose last bits lie below 2^-133).  Of the nine products three are left out, m l, l m and l l, which together are
// within 2^-25 of the product: less than one rounding of an fp32 product.  The products of the high parts have an accumulator
// of their own, the five small ones share another, both start from zero for every 16 columns (rows, positions), and ordinary
// fp32 adds take them to the running total: what the tensor pipe cuts off a sum it accumulates stays small.  2-norm error
// against 64 bits, 16384 positions of 2048 -> (16, 32, 1), gradient at x / of the weights: 2.76e-7 / 2.63e-7 with two TF32 parts
// and three products in one accumulator, 2.11e-7 / 2.29e-7 with fp32 multiply-adds, 1.63e-7 / 1.86e-7 here.
// A NaN stays a NaN in the high part; an infinity becomes one (its remainder is infinity - infinity).
//
// Fragments of mma.m16n8k16 (lane = 4 g + t), two bf16 per register, the first in the low half: A (16 x 16) a0 (g, 2 t + {0, 1})
// a1 (g + 8, 2 t + {0, 1}) a2 (g, 2 t + 8 + {0, 1}) a3 (g + 8, 2 t + 8 + {0, 1}); B (16 x 8) b0 (2 t + {0, 1}, g)
// b1 (2 t + 8 + {0, 1}, g); C (16 x 8) c0 (g, 2 t) c1 (g, 2 t + 1) c2 (g + 8, 2 t) c3 (g + 8, 2 t + 1).  m16n8k8 has a0, a1
// and b0 only.  Which column of x an index of a fragment stands for is free, and chosen so that a lane always moves four
// neighbouring columns.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "bulk_copy.cuh"
#include "kernels_dense.cuh"

namespace b200 {

// Two values into their parts: each register holds the part of `a` in its low half, of `b` in its high half.
__device__ __forceinline__ uint32_t bf16_pair(float a, float b) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    return r;
}
__device__ __forceinline__ float bf16_lo(uint32_t pair) { return __uint_as_float(pair << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t pair) { return __uint_as_float(pair & 0xffff0000u); }
struct Split {
    uint32_t h, m, l;
};
__device__ __forceinline__ Split bf16_split(float a, float b) {
    Split s;
    s.h = bf16_pair(a, b);
    a -= bf16_lo(s.h), b -= bf16_hi(s.h);
    s.m = bf16_pair(a, b);
    s.l = bf16_pair(a - bf16_lo(s.m), b - bf16_hi(s.m));
    return s;
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[2], const uint32_t (&b)[1]) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(b[0]));
}
// total += A B, both in parts [high, middle, low]
template <int NA, int NB>
__device__ __forceinline__ void mma_split(float (&total)[4], const uint32_t (&a)[3][NA], const uint32_t (&b)[3][NB]) {
    float high[4] = {0.f, 0.f, 0.f, 0.f}, rest[4] = {0.f, 0.f, 0.f, 0.f};
    mma_bf16(high, a[0], b[0]);
    mma_bf16(rest, a[1], b[1]);
    mma_bf16(rest, a[0], b[2]);
    mma_bf16(rest, a[2], b[0]);
    mma_bf16(rest, a[0], b[1]);
    mma_bf16(rest, a[1], b[0]);
#pragma unroll
    for (int e = 0; e < 4; e++) total[e] += high[e] + rest[e];
}

constexpr int kMmaCols = 16;  // columns of x in one group of the forward and of dx
template <int M1>
__host__ __device__ constexpr int mma_tiles() { return M1 >= 8 ? M1 / 8 : 1; }  // 8-row tiles (a layer of four rows fills half of one)
constexpr int kTileWords = 32 * 6;  // 32-bit words of 16 columns of an 8-row tile, three parts
// rows that the gradient at x contracts in one step
__host__ __device__ constexpr int dx_rows(int M1) { return M1 >= 16 ? 16 : 8; }
// Words of one fragment table.  Forward, B with (k = column, n = row): [bucket][16-column group][8-row tile], of each lane
// (h0, h1, m0, m1), then of each (l0, l1); its columns are 16 group + 4 t + 0..3 in the order of the pairs, its row is
// 8 tile + g.  Gradient at x, B with (k = row, n = column): [bucket][group][step of dx_rows][part], of each lane the registers
// of columns j = 0, 1: column 16 group + 4 (g / 2) + 2 j + g % 2, rows of the step 4 t + 0..3 in the order of the pairs (16 a
// step) or 2 t + 0, 1 (8 a step).
__host__ __device__ inline size_t mma_table_words(int K1, int O, int M1) {
    return (size_t)O * ((K1 + kMmaCols - 1) / kMmaCols) * (M1 >= 8 ? M1 / 8 : 1) * kTileWords;
}
__device__ __forceinline__ uint32_t split_part(const Split& s, int part) { return part == 0 ? s.h : part == 1 ? s.m : s.l; }

// Weights of one column and four neighbouring rows (k, row .. row + 3) into both tables.
__device__ __forceinline__ void store_fragments(uint32_t* fwd, uint32_t* dxt, int K1, int M1, int k, int col, int row, float4 w) {
    const int groups = (K1 + kMmaCols - 1) / kMmaCols, tiles = M1 >= 8 ? M1 / 8 : 1, c = col & 15;
    const size_t at = ((size_t)k * groups + (col >> 4)) * tiles * kTileWords;
    const Split a = bf16_split(w.x, w.y), b = bf16_split(w.z, w.w);
    uint16_t* f = reinterpret_cast<uint16_t*>(fwd + at + (row >> 3) * kTileWords);
    const int t = c >> 2, pair = (c & 3) >> 1, half = c & 1;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int lane = 4 * ((row + i) & 7) + t;
        const Split& s = i < 2 ? a : b;
        f[(lane * 4 + pair) * 2 + half] = (uint16_t)(i & 1 ? s.h >> 16 : s.h);
        f[(lane * 4 + 2 + pair) * 2 + half] = (uint16_t)(i & 1 ? s.m >> 16 : s.m);
        f[(128 + lane * 2 + pair) * 2 + half] = (uint16_t)(i & 1 ? s.l >> 16 : s.l);
    }
    const int g = 2 * (c >> 2) + (c & 1), j = (c & 3) >> 1;
#pragma unroll
    for (int part = 0; part < 3; part++) {
        const uint32_t lo = split_part(a, part), hi = split_part(b, part);
        if (M1 >= 16) {
            uint32_t* d = dxt + at + (row >> 4) * 2 * kTileWords + part * 128 + (4 * g + ((row & 15) >> 2)) * 4 + 2 * j;
            *reinterpret_cast<uint2*>(d) = make_uint2(lo, hi);
        } else {
            uint32_t* d = dxt + at + part * 64 + (4 * g + (row >> 1)) * 2 + j;
            d[0] = lo, d[2] = hi;
        }
    }
}

// Rebuilds both fragment tables from l1w [column][bucket][row]: a thread per column and four rows, those past the last
// (a layer of four rows fills half a tile, the last group of columns may be short) as zeros.
static __global__ void __launch_bounds__(256) dense_fragments_kernel(const float* __restrict__ W1, uint32_t* __restrict__ fwd, uint32_t* __restrict__ dxt,
                                                                    int K1, int O, int M1) {
    const int cols = (K1 + kMmaCols - 1) / kMmaCols * kMmaCols, quads = M1 >= 8 ? M1 / 4 : 2, total = O * cols * quads;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const int row = i % quads * 4, col = i / quads % cols, k = i / (quads * cols);
        const bool in = row < M1 && col < K1;
        const float4 w = in ? *reinterpret_cast<const float4*>(W1 + (size_t)col * (O * M1) + k * M1 + row) : make_float4(0, 0, 0, 0);
        store_fragments(fwd, dxt, K1, M1, k, col, row, w);
    }
}

// What tile `i` holds: its count (0 past the last), this lane's position in it and its output bucket.  The three look-ups
// depend on one another, so they run three tiles ahead, one a tile.
struct TileAhead {
    int2 t;
    int pos, bucket;
};
struct TileLookup {
    const DenseArgs& a;
    int lane, last;  // (this lane's place in a tile)
    TileAhead ahead[3];
    __device__ void range(TileAhead& s, int i) const { s.t = i < last ? dense_tile_at(a.tiles, i, a.n) : make_int2(0, 0); }
    __device__ void place(TileAhead& s) const { s.pos = s.t.y > 0 ? dense_order_at(a.order, s.t.x + min(lane, s.t.y - 1)) : 0; }
    __device__ void bucket(TileAhead& s) const { s.bucket = s.t.y > 0 && a.O > 1 ? a.buckets[s.pos] : 0; }
    __device__ TileLookup(const DenseArgs& args, int lane_, int first, int last_) : a(args), lane(lane_), last(last_) {
        for (int i = 0; i < 3; i++) range(ahead[i], first + i);
        place(ahead[0]), place(ahead[1]);
        bucket(ahead[0]);
    }
    __device__ TileAhead next(int i) {  // tile i, in turn
        const TileAhead now = ahead[0];
        ahead[0] = ahead[1], ahead[1] = ahead[2];
        range(ahead[2], i + 3);
        bucket(ahead[0]);
        place(ahead[1]);
        return now;
    }
};
// full and empty barriers of a ring of stages, and a walk over them
template <int STAGES>
struct Ring {
    uint64_t full[STAGES], empty[STAGES];
    __device__ void init(int readers) {
        for (int s = 0; s < STAGES; s++) mbar_init(&full[s], 1), mbar_init(&empty[s], readers);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
};
template <int STAGES>
struct RingPlace {
    int slot = 0;
    uint32_t phase = 0;
    __device__ void advance() {
        if (++slot == STAGES) slot = 0, phase ^= 1;
    }
};
__host__ __device__ constexpr int dense_mma_ctas(int M1) { return M1 > 16 ? 1 : 2; }
__device__ __forceinline__ void copy16_async(void* smem_dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem_dst)), "l"(src) : "memory");
}

// First layer, forward: sums of slices of the columns, partial[part][tile][32][M1].  A CTA keeps one bucket's fragments of a
// slice of kSliceCols columns in shared memory and walks a run of tiles (up to 32 positions of one output bucket each); a warp
// takes a tile by itself, every lane four 16-byte pieces of x (rows g, g + 8, g + 16, g + 24) of each 16-column group.  A
// lane copies its pieces into its own places of a ring (cp.async), four groups ahead of the products and across the tiles'
// ends, so that no warp waits for another; the look-ups (range, positions, bucket) run a tile ahead of the copies.
// With few tiles `split` warps share a slice of one.  The layers behind, and the sum of the parts, have a kernel of their own:
// they keep a CTA's loads from flowing, and the weights read from L2 for every tile (as much as x) cost 75 us at 131072.
// At 131072 positions (K1 = 2048, M1 = 16) 0.400 ms for both kernels' work in one, a CTA per tile with x loaded into registers;
// now 0.249 + 0.060 from a cold cache, 0.337 for both in a step (this kernel with two TF32 parts: 0.228), against 0.165 for
// reading x at the copy rate; at 16384 0.060.
// grid = (slices, runs), block = 256, dynamic shared memory = dense_mma_smem<M1>().
constexpr int kSliceCols = 256, kFwdDepth = 5, kFwdAhead = 8;
template <int M1>
__host__ __device__ constexpr size_t dense_mma_smem() {
    return ((size_t)kFwdDepth * 4 * 256 * sizeof(float4) + (size_t)kSliceCols / kMmaCols * mma_tiles<M1>() * kTileWords * 4);
}

template <int M1>
__global__ void __launch_bounds__(256, dense_mma_ctas(M1)) dense_first_mma_kernel(const __grid_constant__ DenseArgs a, int split) {
    constexpr int NT = mma_tiles<M1>(), kGroups = kSliceCols / kMmaCols;
    extern __shared__ __align__(16) float dense_smem[];  // [stage][row of four][thread] float4, then the slice's fragments
    __shared__ int4 s_units[8][kFwdAhead];  // per warp, of the units between its copies and its products: range, bucket
    static_assert(kFwdAhead > kFwdDepth, "units of one group each");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
    const int slice = blockIdx.x, groups = (a.K1 + kMmaCols - 1) / kMmaCols, slice_groups = min(kGroups, groups - slice * kGroups);
    const int per_unit = kGroups / split;
    // units = tiles x split; a CTA's run of them is dealt to its warps in turn
    const int run0 = (int)((long long)a.ntiles * split * blockIdx.y / gridDim.y), run1 = (int)((long long)a.ntiles * split * (blockIdx.y + 1) / gridDim.y);
    float4* ring = reinterpret_cast<float4*>(dense_smem) + threadIdx.x;
    uint32_t* s_w = reinterpret_cast<uint32_t*>(dense_smem) + kFwdDepth * 4 * 256 * 4;

    // The copies' side: rows and range of the unit being copied, positions of the next one, range of the one after that.
    auto range = [&](int unit) { return unit < run1 ? dense_tile_at(a.tiles, unit / split, a.n) : make_int2(0, 0); };
    int next_pos[4];
    auto places = [&](int2 t) {
#pragma unroll
        for (int r = 0; r < 4; r++) next_pos[r] = t.y > 0 ? dense_order_at(a.order, t.x + min(g + 8 * r, t.y - 1)) : 0;
    };
    const float* row[4];
    int copy_unit = run0 + warp, copy_group = copy_unit % split * per_unit, copy_stage = 0, copy_bucket = 0;
    int2 copy_range = range(copy_unit), next_range = range(copy_unit + 8), after_next = range(copy_unit + 16);
    bool told = false;
    auto enter = [&]() {  // the copies reach copy_unit, whose positions are in next_pos
#pragma unroll
        for (int r = 0; r < 4; r++) row[r] = a.x + (size_t)next_pos[r] * a.K1 + slice * kSliceCols + 4 * t4;
        copy_bucket = a.O > 1 && copy_range.y > 0 ? a.buckets[__shfl_sync(0xffffffffu, next_pos[0], 0)] : 0;
        told = false;  // (told a group later, when the bucket has arrived)
        places(next_range);
    };
    auto copy = [&]() {  // one group, and on to the next
        if (!told) {
            if (lane == 0) s_units[warp][copy_unit >> 3 & (kFwdAhead - 1)] = make_int4(copy_range.x, copy_range.y, copy_bucket, 0);
            told = true;
        }
        if (copy_range.y > 0) {
            if (slice * kSliceCols + copy_group * kMmaCols + 4 * t4 < a.K1)  // K1 is a multiple of four: a piece is inside or outside
#pragma unroll
                for (int r = 0; r < 4; r++) copy16_async(ring + (copy_stage * 4 + r) * 256, row[r] + copy_group * kMmaCols);
            copy_stage = copy_stage + 1 < kFwdDepth ? copy_stage + 1 : 0;
            if (++copy_group % per_unit == 0 || copy_group >= slice_groups) {
                copy_unit += 8;
                copy_group = copy_unit % split * per_unit;
                copy_range = next_range, next_range = after_next, after_next = range(copy_unit + 16);
                enter();
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    places(copy_range);
    enter();
    // the bucket of a round's first unit, looked up like the rows
    auto lead_pos = [&](int2 t) { return t.y > 0 ? dense_order_at(a.order, t.x) : -1; };
    auto lead_bucket = [&](int pos) { return pos < 0 ? -1 : a.O > 1 ? a.buckets[pos] : 0; };
    int bucket0 = lead_bucket(lead_pos(range(run0))), pos1 = lead_pos(range(run0 + 8));
    int2 range2 = range(run0 + 16);
    int held = -1, stage = 0;  // the bucket whose fragments are in shared memory
    auto hold = [&](int bucket) {
        const uint4* table = reinterpret_cast<const uint4*>(a.W1f + ((size_t)bucket * groups + slice * kGroups) * NT * kTileWords);
        for (int i = threadIdx.x; i < slice_groups * NT * (kTileWords / 4); i += 256) reinterpret_cast<uint4*>(s_w)[i] = __ldg(table + i);
        held = bucket;
    };
    if (bucket0 >= 0) hold(bucket0);
    step_begin(a.stamp);  // everything so far was there before the kernel before this one began
#pragma unroll 1
    for (int i = 0; i < kFwdDepth - 1; i++) copy();
    __syncthreads();
    for (int round = run0; round < run1; round += 8) {
        const int unit = round + warp;
        const int wanted = bucket0;
        if (wanted < 0) break;  // (uniform; the launch is sized from the batch size alone, empty tiles come last)
        bucket0 = lead_bucket(pos1), pos1 = lead_pos(range2), range2 = range(round + 24);
        if (wanted != held) {
            __syncthreads();
            hold(wanted);
            __syncthreads();
        }
        if (unit >= run1) continue;
        __syncwarp();
        const int4 at = s_units[warp][unit >> 3 & (kFwdAhead - 1)];
        if (at.y <= 0) continue;
        const int first = unit % split * per_unit, last = min(first + per_unit, slice_groups);
        // (a tile of the next bucket that shares a round with tiles of this one reads the fragments where they are)
        const uint32_t* table = at.z == held ? s_w : a.W1f + ((size_t)at.z * groups + slice * kGroups) * NT * kTileWords;
        float acc[2][NT][4];
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int nt = 0; nt < NT; nt++)
#pragma unroll
                for (int e = 0; e < 4; e++) acc[m][nt][e] = 0.f;
#pragma unroll 1
        for (int group = first; group < last; group++) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kFwdDepth - 2) : "memory");
            const bool in = slice * kSliceCols + group * kMmaCols + 4 * t4 < a.K1;
            float4 xs[4];
            uint32_t w[NT][3][2];
#pragma unroll
            for (int r = 0; r < 4; r++) xs[r] = in ? ring[(stage * 4 + r) * 256] : make_float4(0, 0, 0, 0);
#pragma unroll
            for (int nt = 0; nt < NT; nt++) {
                const uint32_t* tile = table + (group * NT + nt) * kTileWords;
                const uint4 hm = *reinterpret_cast<const uint4*>(tile + 4 * lane);
                const uint2 l = *reinterpret_cast<const uint2*>(tile + 128 + 2 * lane);
                w[nt][0][0] = hm.x, w[nt][0][1] = hm.y, w[nt][1][0] = hm.z, w[nt][1][1] = hm.w, w[nt][2][0] = l.x, w[nt][2][1] = l.y;
            }
            stage = stage + 1 < kFwdDepth ? stage + 1 : 0;
            copy();
#pragma unroll
            for (int m = 0; m < 2; m++) {
                uint32_t xp[3][4];
#pragma unroll
                for (int e = 0; e < 4; e++) {  // rows g and g + 8 of the half, first and second pair of columns
                    const float4 v = xs[2 * m + (e & 1)];
                    const Split s = e < 2 ? bf16_split(v.x, v.y) : bf16_split(v.z, v.w);
                    xp[0][e] = s.h, xp[1][e] = s.m, xp[2][e] = s.l;
                }
#pragma unroll
                for (int nt = 0; nt < NT; nt++) mma_split(acc[m][nt], xp, w[nt]);
            }
        }
        float* partial = a.partial + ((size_t)(slice * split + unit % split) * a.ntiles + unit / split) * kDenseTile * M1;
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int nt = 0; nt < NT; nt++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int p = 16 * m + g + 8 * h, r = 8 * nt + 2 * t4;
                    if (r < M1 && p < at.y) *reinterpret_cast<float2*>(partial + p * M1 + r) = make_float2(acc[m][nt][2 * h], acc[m][nt][2 * h + 1]);
                }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// words before step `i` (16 places of a tile) of the weight gradient's operand: [step][16-row tile][part][lane] uint4, rows r = 16
// tile + g (+ 8), places of the step 2 t + {0, 1} (+ 8)
constexpr int kWgradStep = 16;
template <int M1>
__host__ __device__ constexpr size_t wgrad_table_words(size_t i) { return i * (M1 > 16 ? M1 / 16 : 1) * 384; }

// The rest of the forward: sum of the first layer's parts, small layers, loss, the way back to the first layer's
// pre-activation gradient (also as the operand of its weight gradient), weight gradients of the small layers and the first
// layer's bias gradient (kept in registers until the bucket changes).  A CTA takes a
// run of tiles, a warp eight of a tile's 32 positions: four lanes per position, each with a quarter of the second layer's 32
// rows (zero past the last); for the weight gradients a lane is a row.  Bound by latency: 60 us at 131072 positions
// (64 MB of parts), 17 at 16384, from a cold cache.
// grid = up to kSmallCtas per SM, block = 128.
constexpr int kSmallThreads = 128, kSmallCtas = 4;
template <int M1>
__global__ void __launch_bounds__(kSmallThreads, M1 > 16 ? 2 : 4) dense_small_mma_kernel(const __grid_constant__ DenseArgs a, int parts) {
    constexpr int kRow = M1 + 4, kPer = M1 / 4;   // M1 columns in pieces of four; each of a position's lanes sums kPer of a1
    __shared__ __align__(16) float s_w2[32 * M1 + 16];     // [row][column], four floats further every eight rows: a quarter each, no two in one bank
    __shared__ float s_b1[M1], s_b2[32], s_w3[32], s_bias3;
    __shared__ __align__(16) float s_a1[4][8][kRow];
    __shared__ float s_dz2[4][8][33], s_a2[4][8][33], s_dout[4][8], s_own[4][M1 + 2][32], s_own1[4][M1], s_own_bias[4];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, p = lane >> 2, quarter = lane & 3;
    const int M2 = a.M[1], OM2 = a.O * M2;
    const int first = (int)((long long)a.ntiles * blockIdx.x / gridDim.x), last = (int)((long long)a.ntiles * (blockIdx.x + 1) / gridDim.x);
    float own1[kPer], own[M1 + 1], own3 = 0.f, own3_bias = 0.f, my_loss = 0.f;  // this lane's row of the second layer: its columns, its bias; the third layer
#pragma unroll
    for (int c = 0; c <= M1; c++) own[c] = 0.f;
#pragma unroll
    for (int i = 0; i < kPer; i++) own1[i] = 0.f;
    int cur = -1;
    auto flush = [&]() {
        if (cur < 0 || !a.want_grad) return;  // (uniform) the four warps' sums, then one addition per CTA
#pragma unroll
        for (int c = 0; c <= M1; c++) s_own[warp][c][lane] = own[c];
        s_own[warp][M1 + 1][lane] = own3;
        own3_bias = warp_sum(own3_bias);
        if (lane == 0) s_own_bias[warp] = own3_bias;
#pragma unroll
        for (int i = 0; i < kPer; i++) {
#pragma unroll
            for (int d = 4; d < 32; d <<= 1) own1[i] += __shfl_xor_sync(0xffffffffu, own1[i], d);
            if (p == 0) s_own1[warp][kPer * quarter + i] = own1[i];
            own1[i] = 0.f;
        }
        __syncthreads();
        if ((int)threadIdx.x < M1) atomicAdd(a.gB[0] + cur * M1 + threadIdx.x, (s_own1[0][threadIdx.x] + s_own1[1][threadIdx.x]) + (s_own1[2][threadIdx.x] + s_own1[3][threadIdx.x]));
        for (int c = warp; c < M1 + 2; c += 4) {
            const float sum = (s_own[0][c][lane] + s_own[1][c][lane]) + (s_own[2][c][lane] + s_own[3][c][lane]);
            if (lane < M2 && (c <= M1 || a.n_dense == 3) && sum != 0.f)
                atomicAdd(c < M1 ? a.gW[1] + (size_t)c * OM2 + cur * M2 + lane : c == M1 ? a.gB[1] + cur * M2 + lane : a.gW[2] + (size_t)lane * a.O + cur, sum);
        }
        if (threadIdx.x == 0 && a.n_dense == 3) atomicAdd(a.gB[2] + cur, (s_own_bias[0] + s_own_bias[1]) + (s_own_bias[2] + s_own_bias[3]));
#pragma unroll
        for (int c = 0; c <= M1; c++) own[c] = 0.f;
        own3 = own3_bias = 0.f;
    };
    const int at = 8 * warp + p;
    auto hold = [&](int k) {  // a bucket's small layers, zero past their rows
        cur = k;
        for (int i = threadIdx.x; i < 32 * M1; i += kSmallThreads) {
            const int r = i & 31, c = i >> 5;
            s_w2[r * M1 + c + 4 * (r >> 3)] = r < M2 ? a.W[1][c * OM2 + k * M2 + r] : 0.f;
        }
        if (warp == 0) {
            s_b2[lane] = lane < M2 ? a.B[1][k * M2 + lane] : 0.f;
            s_w3[lane] = lane < M2 && a.n_dense == 3 ? a.W[2][lane * a.O + k] : 0.f;
            if (lane < M1) s_b1[lane] = a.B[0][k * M1 + lane];
            if (lane == 0) s_bias3 = a.n_dense == 3 ? a.B[2][k] : 0.f;
        }
    };
    TileLookup lookup(a, at, first, last);
    if (lookup.ahead[0].t.y > 0) hold(lookup.ahead[0].bucket);
    step_begin(nullptr);  // everything so far was there before the kernel before this one began
    __syncthreads();
    for (int tile = first; tile < last; tile++) {
        const TileAhead now = lookup.next(tile);
        const int2 t = now.t;
        if (t.y <= 0) break;
        const bool on = at < t.y;
        const int pos = now.pos, k = now.bucket;
        const float target = a.want_grad ? a.targets[pos] : 0.f;
        float z1[kPer];
#pragma unroll
        for (int i = 0; i < kPer; i++) z1[i] = 0.f;
        {
            const float* src = a.partial + ((size_t)tile * kDenseTile + min(at, t.y - 1)) * M1 + kPer * quarter;
#pragma unroll 8
            for (int w = 0; w < parts; w++, src += (size_t)a.ntiles * kDenseTile * M1)
                if constexpr (kPer >= 4) {
#pragma unroll
                    for (int i = 0; i < kPer; i += 4) {
                        const float4 v = *reinterpret_cast<const float4*>(src + i);
                        z1[i] += v.x, z1[i + 1] += v.y, z1[i + 2] += v.z, z1[i + 3] += v.w;
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < kPer; i++) z1[i] += src[i];
                }
        }
        if (k != cur) {
            flush();
            __syncthreads();
            hold(k);
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < kPer; i++) s_a1[warp][p][kPer * quarter + i] = on ? act_fwd(a.act[0], z1[i] + s_b1[kPer * quarter + i]) : 0.f;
        __syncwarp();
        float a1[M1];
#pragma unroll
        for (int c = 0; c < M1; c += 4) {
            const float4 v = *reinterpret_cast<const float4*>(&s_a1[warp][p][c]);
            a1[c] = v.x, a1[c + 1] = v.y, a1[c + 2] = v.z, a1[c + 3] = v.w;
        }
        const float* w2 = s_w2 + quarter * (8 * M1 + 4);
        float* y2 = &s_a2[warp][p][8 * quarter];  // outputs of the second layer's rows 8 quarter + i
        float o = 0.f;
#pragma unroll 2
        for (int i = 0; i < 8; i++) {
            float z = 0.f;
#pragma unroll
            for (int c = 0; c < M1; c += 4) {
                const float4 w = *reinterpret_cast<const float4*>(w2 + i * M1 + c);
                z += w.x * a1[c];
                z += w.y * a1[c + 1];
                z += w.z * a1[c + 2];
                z += w.w * a1[c + 3];
            }
            z += s_b2[8 * quarter + i];
            const float y = a.n_dense == 2 ? z : 8 * quarter + i < M2 ? act_fwd(a.act[1], z) : 0.f;
            y2[i] = y;
            o += s_w3[8 * quarter + i] * y;
        }
        if (a.n_dense == 2) {
            o = __shfl_sync(0xffffffffu, y2[0], lane & ~3);  // (of the position's first lane)
        } else {
            o += __shfl_xor_sync(0xffffffffu, o, 1);
            o += __shfl_xor_sync(0xffffffffu, o, 2);
            o += s_bias3;
        }
        if (on && quarter == 0) {
            a.out[pos] = o;
            if (a.out_host) a.out_host[pos] = o;
        }
        if (!a.want_grad) continue;
        const float s = 1.f / (1.f + expf(-o));
        const float diff = s - target;
        if (on && quarter == 0) my_loss += diff * diff;
        const float dout = on ? (diff + diff) * (s * (1.f - s)) : 0.f;
        if (quarter == 0) s_dout[warp][p] = dout;
        float dz1[M1];
#pragma unroll
        for (int c = 0; c < M1; c++) dz1[c] = 0.f;
#pragma unroll 2
        for (int i = 0; i < 8; i++) {  // gradient at the second layer's pre-activation, and what it gives the first
            const int r = 8 * quarter + i;
            const float d = a.n_dense == 2 ? (r == 0 ? dout : 0.f) : r < M2 ? (s_w3[r] * dout) * act_bwd(a.act[1], y2[i]) : 0.f;
            s_dz2[warp][p][r] = d;
#pragma unroll
            for (int c = 0; c < M1; c += 4) {
                const float4 w = *reinterpret_cast<const float4*>(w2 + i * M1 + c);
                dz1[c] += w.x * d, dz1[c + 1] += w.y * d, dz1[c + 2] += w.z * d, dz1[c + 3] += w.w * d;
            }
        }
        // the sums of the four lanes of a position: each is left with its kPer columns
        float mine[kPer];
        if (M1 >= 8) {
            const bool upper = quarter & 2, odd = quarter & 1;
#pragma unroll
            for (int c = 0; c < M1 / 2; c++) {
                const float give = upper ? dz1[c] : dz1[c + M1 / 2], keep = upper ? dz1[c + M1 / 2] : dz1[c];
                dz1[c] = keep + __shfl_xor_sync(0xffffffffu, give, 2);
            }
#pragma unroll
            for (int c = 0; c < kPer; c++) {
                const float give = odd ? dz1[c] : dz1[c + kPer], keep = odd ? dz1[c + kPer] : dz1[c];
                mine[c] = keep + __shfl_xor_sync(0xffffffffu, give, 1);
            }
        } else {
#pragma unroll
            for (int c = 0; c < M1; c++) {
                dz1[c] += __shfl_xor_sync(0xffffffffu, dz1[c], 1);
                dz1[c] += __shfl_xor_sync(0xffffffffu, dz1[c], 2);
            }
            mine[0] = quarter == 0 ? dz1[0] : quarter == 1 ? dz1[1] : quarter == 2 ? dz1[2] : dz1[3];
        }
#pragma unroll
        for (int i = 0; i < kPer; i++) {
            const int r = kPer * quarter + i;
            const float d = on ? mine[i] * act_bwd(a.act[0], s_a1[warp][p][r]) : 0.f;
            if (on) a.dz[0][(size_t)pos * M1 + r] = d;
            own1[i] += d;
            // A of the weight gradient: the lane of an even place stores its own and its neighbour's
            const float next = __shfl_xor_sync(0xffffffffu, d, 4);
            if (!(p & 1)) {
                const Split pair = bf16_split(d, next);
                const int q = at & (kWgradStep - 1);
                uint32_t* out = a.dz_frag + wgrad_table_words<M1>((size_t)tile * 2 + (at >> 4)) + (r >> 4) * 384 + (4 * (r & 7) + ((q & 7) >> 1)) * 4 + (r >> 3 & 1) + 2 * (q >> 3);
                out[0] = pair.h, out[128] = pair.m, out[256] = pair.l;
            }
        }
        __syncwarp();
#pragma unroll 4
        for (int q = 0; q < 8; q++) {  // layer 2: X = a1, dY = dz2; layer 3: X = a2, dY = dout (one row)
            const float d = s_dz2[warp][q][lane];
#pragma unroll
            for (int c = 0; c < M1; c += 4) {
                const float4 v = *reinterpret_cast<const float4*>(&s_a1[warp][q][c]);
                own[c] += d * v.x, own[c + 1] += d * v.y, own[c + 2] += d * v.z, own[c + 3] += d * v.w;
            }
            own[M1] += d;
            own3 += s_dout[warp][q] * s_a2[warp][q][lane];
        }
        if (lane < 8) own3_bias += s_dout[warp][lane];
        __syncwarp();
    }
    flush();
    if (a.want_grad) {
        my_loss = warp_sum(my_loss);
        __syncthreads();
        if (lane == 0) s_own_bias[warp] = my_loss;
        __syncthreads();
        if (threadIdx.x == 0) atomicAdd(a.loss, (s_own_bias[0] + s_own_bias[1]) + (s_own_bias[2] + s_own_bias[3]));
    }
}


// dx[b][c] = sum_r W1[c][k_b][r] * dz1[b][r]   (Matmul::backward, matmul.rs:99-126, on the selected rows).  Same tiles; a
// warp keeps the split gradients of all 32 positions in registers and walks the 16-column groups, storing four neighbouring
// columns per lane and row.  With fp32 multiply-adds this and the weight
// gradient took 0.681 ms at 131072 positions, K1 = 2048, M1 = 16; now 0.229 here (0.165 for writing dx at the copy rate).
// grid = ntiles, block = 256.
template <int M1>
__global__ void __launch_bounds__(256, (M1 > 16 ? 1 : 2)) dense_dx_mma_kernel(DenseArgs a, float* dx) {
    step_begin(a.stamp);
    constexpr int S = M1 >= 16 ? M1 / 16 : 1, NA = M1 >= 16 ? 4 : 2, NB = NA / 2;  // steps; registers of a part of A and of one column tile of B
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
    const int2 t = dense_tile_at(a.tiles, blockIdx.x, a.n);
    if (t.y <= 0) return;
    const int groups = (a.K1 + kMmaCols - 1) / kMmaCols;
    float* row[4];
    uint32_t dz[2][S][3][NA];
    int k = 0;
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const int pos = dense_order_at(a.order, t.x + min(g + 8 * r, t.y - 1));
        if (r == 0) k = a.buckets[pos];
        row[r] = dx + (size_t)pos * a.K1 + 4 * t4;
        const float* own = a.dz[0] + (size_t)pos * M1;
#pragma unroll
        for (int s = 0; s < S; s++) {
            auto put = [&](int e, Split v) { dz[r >> 1][s][0][e] = v.h, dz[r >> 1][s][1][e] = v.m, dz[r >> 1][s][2][e] = v.l; };
            if constexpr (NA == 4) {
                const float4 v = *reinterpret_cast<const float4*>(own + 16 * s + 4 * t4);
                put(r & 1, bf16_split(v.x, v.y));
                put((r & 1) + 2, bf16_split(v.z, v.w));
            } else {
                float2 v = make_float2(0.f, 0.f);
                if (2 * t4 < M1) v = *reinterpret_cast<const float2*>(own + 2 * t4);
                put(r & 1, bf16_split(v.x, v.y));
            }
        }
    }
    const uint32_t* table = a.W1d + (size_t)k * groups * S * (NB * kTileWords) + lane * 2 * NB;
    uint32_t ahead[S][3][2 * NB];  // [step][part][column tile, register]
    auto fetch = [&](int grp) {
        if (grp < groups)
#pragma unroll
            for (int s = 0; s < S; s++)
#pragma unroll
                for (int part = 0; part < 3; part++) {
                    const uint32_t* src = table + (size_t)(grp * S + s) * (NB * kTileWords) + part * 64 * NB;
                    if constexpr (NB == 2) {
                        const uint4 v = __ldg(reinterpret_cast<const uint4*>(src));
                        ahead[s][part][0] = v.x, ahead[s][part][1] = v.y, ahead[s][part][2] = v.z, ahead[s][part][3] = v.w;
                    } else {
                        const uint2 v = __ldg(reinterpret_cast<const uint2*>(src));
                        ahead[s][part][0] = v.x, ahead[s][part][1] = v.y;
                    }
                }
    };
    fetch(warp);
    unsigned largest = 0;
    for (int grp = warp; grp < groups; grp += 8) {
        uint32_t b[S][2][3][NB];
#pragma unroll
        for (int s = 0; s < S; s++)
#pragma unroll
            for (int j = 0; j < 2; j++)
#pragma unroll
                for (int part = 0; part < 3; part++)
#pragma unroll
                    for (int e = 0; e < NB; e++) b[s][j][part][e] = ahead[s][part][NB * j + e];
        fetch(grp + 8);
        const bool in = grp * kMmaCols + 4 * t4 < a.K1;
#pragma unroll
        for (int m = 0; m < 2; m++) {
            float c[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
            for (int s = 0; s < S; s++)
#pragma unroll
                for (int j = 0; j < 2; j++) mma_split(c[j], dz[m][s], b[s][j]);
#pragma unroll
            for (int h = 0; h < 2; h++)
                if (in && 16 * m + 8 * h + g < t.y) {
                    *reinterpret_cast<float4*>(row[2 * m + h] + grp * kMmaCols) = make_float4(c[0][2 * h], c[0][2 * h + 1], c[1][2 * h], c[1][2 * h + 1]);
                    largest = max(max(largest, max(magnitude(c[0][2 * h]), magnitude(c[0][2 * h + 1]))), max(magnitude(c[1][2 * h]), magnitude(c[1][2 * h + 1])));
                }
        }
    }
    raise_magnitude(a.gmax, largest);
}

// Weight gradient of the first layer: gW[c][k][r] += sum_b [k_b == k] dz1[b][r] * x[b][c].  Positions contract, sixteen
// a step; r is the M of the product and columns its N: a lane takes four neighbouring columns of four positions, and value j
// of each belongs to column tile j.  A warp owns 64 columns (two groups of 32), the eight of a CTA 512; the CTA walks a
// run of dense tiles, of which a ninth warp copies sixteen rows of x and their dz1 (fragments that the small layers' kernel has
// written in the order of the tiles) at a time into a ring of stages, and adds its sums to the gradient when the output bucket
// changes.  (x loaded into registers and dz1 split through shared memory a tile at a time, with two barriers: 0.365 ms at
// 131072 positions, K1 = 2048, M1 = 16; lanes copying their own pieces by cp.async, as the forward does: 0.370; this: 0.244
// from a cold cache (0.240 with two TF32 parts and eight positions a step), against 0.165 for reading x at the copy rate.  A
// bulk copy costs the warp that issues it 70 to 100 clocks, so it should be long.)
// grid = (ceil(K1 / 512), runs), block = 288, dynamic shared memory = wgrad_smem<M1>().
constexpr int kRingThreads = 288;
constexpr int kWgradCols = 64, kWgradStages = 3;
constexpr int kWgradPitch = 8 * kWgradCols + 4;  // (rows 2 t of a step, four banks and eight apart: no two lanes of a load in one bank)
template <int M1>
__host__ __device__ constexpr int wgrad_stage_floats() { return kWgradStep * kWgradPitch + (int)wgrad_table_words<M1>(1); }
template <int M1>
__host__ __device__ constexpr size_t wgrad_smem() { return (size_t)kWgradStages * wgrad_stage_floats<M1>() * sizeof(float); }

template <int M1>
__global__ void __launch_bounds__(kRingThreads, dense_mma_ctas(M1)) dense_wgrad_mma_kernel(const __grid_constant__ DenseArgs a, float* gW) {
    constexpr int MT = M1 > 16 ? M1 / 16 : 1, kTable = (int)wgrad_table_words<M1>(1);
    extern __shared__ __align__(16) float wgrad_smem_raw[];
    __shared__ Ring<kWgradStages> ring;
    __shared__ int s_rows[kWgradStages], s_bucket[kWgradStages];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
    if (threadIdx.x == 0) ring.init(8);
    __syncthreads();
    const int first = (int)((long long)a.ntiles * blockIdx.y / gridDim.y), last = (int)((long long)a.ntiles * (blockIdx.y + 1) / gridDim.y);
    const int cta_col = blockIdx.x * 8 * kWgradCols;
    RingPlace<kWgradStages> at;
    if (warp == 8) {
        TileLookup lookup(a, lane, first, last);
        step_begin(nullptr);  // everything so far was there before the kernel before this one began
        const uint32_t bytes = (uint32_t)min(8 * kWgradCols, a.K1 - cta_col) * 4;
        for (int tile = first;; tile++) {
            const TileAhead now = lookup.next(tile);
            for (int p = 0; p < max(1, now.t.y); p += kWgradStep) {
                const int rows = max(0, min(kWgradStep, now.t.y - p)), pos = __shfl_sync(0xffffffffu, now.pos, (p + lane) & 31);
                if (!mbar_wait(&ring.empty[at.slot], at.phase ^ 1)) return;
                __syncwarp();
                float* stage = wgrad_smem_raw + (size_t)at.slot * wgrad_stage_floats<M1>();
                if (lane == 0) {
                    s_rows[at.slot] = rows;
                    s_bucket[at.slot] = now.bucket;
                    mbar_expect_tx(&ring.full[at.slot], rows ? rows * bytes + kTable * 4 : 0);
                }
                __syncwarp();
                if (lane < rows) bulk_load(stage + lane * kWgradPitch, a.x + (size_t)pos * a.K1 + cta_col, bytes, &ring.full[at.slot]);
                if (lane == kWgradStep && rows)
                    bulk_load(stage + kWgradStep * kWgradPitch, a.dz_frag + wgrad_table_words<M1>((size_t)tile * 2 + p / kWgradStep), kTable * 4, &ring.full[at.slot]);
                at.advance();
            }
            if (now.t.y <= 0) return;  // (the readers stop at a stage without rows)
        }
    }
    step_begin(nullptr);
    const int c0 = cta_col + warp * kWgradCols, OM = a.O * M1;
    float acc[MT][8][4];
    auto clear = [&]() {
#pragma unroll
        for (int m = 0; m < MT; m++)
#pragma unroll
            for (int j = 0; j < 8; j++)
#pragma unroll
                for (int e = 0; e < 4; e++) acc[m][j][e] = 0.f;
    };
    clear();
    int cur = -1;
    auto flush = [&]() {
        if (cur < 0) return;
#pragma unroll
        for (int m = 0; m < MT; m++)
#pragma unroll
            for (int j = 0; j < 8; j++)
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    // tile j of a 32-column group: column index n stands for 4 n + j
                    const int c = c0 + 32 * (j >> 2) + 4 * (2 * t4 + (e & 1)) + (j & 3), r = 16 * m + g + 8 * (e >> 1);
                    if (c < a.K1 && r < M1 && acc[m][j][e] != 0.f) atomicAdd(gW + (size_t)c * OM + cur * M1 + r, acc[m][j][e]);
                }
        clear();
    };
    for (;; at.advance()) {
        if (!mbar_wait(&ring.full[at.slot], at.phase)) {
            *a.gave_up = 1;
            return;
        }
        const int rows = s_rows[at.slot], k = s_bucket[at.slot];
        if (rows == 0) break;
        if (k != cur) {
            flush();
            cur = k;
        }
        const float* stage = wgrad_smem_raw + (size_t)at.slot * wgrad_stage_floats<M1>();
        const uint4* table = reinterpret_cast<const uint4*>(stage + kWgradStep * kWgradPitch) + lane;
        uint32_t dz[MT][3][4];
#pragma unroll
        for (int m = 0; m < MT; m++)
#pragma unroll
            for (int part = 0; part < 3; part++) {
                const uint4 v = table[(3 * m + part) * 32];
                const uint32_t e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int i = 0; i < 4; i++) dz[m][part][i] = 16 * m + 8 * (i & 1) + g < M1 ? e[i] : 0u;  // (the table has no rows past M1)
            }
#pragma unroll
        for (int h = 0; h < 2; h++) {  // the warp's two groups of 32 columns
            const int c = warp * kWgradCols + 32 * h + 4 * g;
            const bool in = cta_col + c < a.K1;
            float4 x[4];  // of four places; those past the last hold what the stage held before, or nothing (their factor is zero)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int place = 2 * t4 + (i & 1) + 8 * (i >> 1);
                x[i] = in && place < rows ? *reinterpret_cast<const float4*>(stage + place * kWgradPitch + c) : make_float4(0, 0, 0, 0);
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                auto col = [&](const float4& v) { return j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w; };
                const Split s0 = bf16_split(col(x[0]), col(x[1])), s1 = bf16_split(col(x[2]), col(x[3]));
                const uint32_t xp[3][2] = {{s0.h, s1.h}, {s0.m, s1.m}, {s0.l, s1.l}};
#pragma unroll
                for (int m = 0; m < MT; m++) mma_split(acc[m][4 * h + j], dz[m], xp);
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&ring.empty[at.slot]);
    }
    flush();
}

}  // namespace b200
