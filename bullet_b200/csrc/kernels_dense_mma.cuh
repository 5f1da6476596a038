// The first dense layer of multi-layer networks (four or more rows per output bucket) on the tensor pipe: forward, gradient at
// its input, weight gradient.
//
// Semantics as in kernels_dense.cuh.  All three are streams over x or dx (K1 floats per position) with a contraction that is
// only M1 wide, so HBM bounds them: 8 KB per position and pass at K1 = 2048.  fp32 multiply-adds could not keep up with it
// (they held the kernels at a third of the copy rate); mma.sync does at a few per cent of its own rate, straight from
// registers, without the staging through shared memory and tensor memory that tcgen05 would add for a 16-wide product.
//
// fp32 operands are split into two TF32 parts, each rounded to nearest: hi keeps 11 bits and lo the next 11, so that hi + lo
// is within 2^-24 of the value; of the four products lo * lo (2^-24 and less of the result) is left out.  A few steps
// accumulate in the tensor pipe, then their sum is added to the running total with an ordinary fp32 add.
//
// Fragments of mma.m16n8k8 (lane = 4 g + t): A (16 x 8) a0 (g, t) a1 (g + 8, t) a2 (g, t + 4) a3 (g + 8, t + 4); B (8 x 8)
// b0 (t, g) b1 (t + 4, g); C (16 x 8) c0 (g, 2 t) c1 (g, 2 t + 1) c2 (g + 8, 2 t) c3 (g + 8, 2 t + 1).  Which column of x an
// index of a fragment stands for is free, and chosen so that a lane always moves four neighbouring columns.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels_dense.cuh"

namespace b200 {

// The tensor pipe reads the upper 19 bits of a TF32 operand, so adding half of the last of them rounds to nearest, ties away
// (cvt.rna.tf32 is several instructions more; it also keeps infinities, which become NaN here: a pass that met one is lost
// either way).
__device__ __forceinline__ void tf32_split(float v, uint32_t& hi, uint32_t& lo) {
    hi = __float_as_uint(v) + 0x1000u;
    lo = __float_as_uint(v - __uint_as_float(hi & 0xffffe000u)) + 0x1000u;
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

constexpr int kMmaCols = 16;  // columns of x in one group of the forward and of dx
template <int M1>
__host__ __device__ constexpr int mma_tiles() { return M1 >= 8 ? M1 / 8 : 1; }  // 8-row tiles (a layer of four rows fills half of one)
// floats of one fragment table: [bucket][16-column group][8-row tile][hi, lo][lane] float4
__host__ __device__ inline size_t mma_table_floats(int K1, int O, int M1) {
    return (size_t)O * ((K1 + kMmaCols - 1) / kMmaCols) * (M1 >= 8 ? M1 / 8 : 1) * 2 * 32 * 4;
}

// Rebuilds both fragment tables from l1w [column][bucket][row] after every update.  `fwd`: B of the forward, (k = column,
// n = row): element (s, i) of a lane's float4 is column 16 grp + 4 t + 2 s + i, row 8 tile + g.  `dxt`: B of dx, (k = row,
// n = column): element (j, i) is column 16 grp + 4 (g / 2) + 2 j + g % 2, row 8 tile + t + 4 i.
static __global__ void __launch_bounds__(256) dense_fragments_kernel(const float* __restrict__ W1, float4* __restrict__ fwd, float4* __restrict__ dxt,
                                                                    int K1, int O, int M1, int tiles) {
    const int groups = (K1 + kMmaCols - 1) / kMmaCols, total = O * groups * tiles * 32;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const int lane = i & 31, tile = (i >> 5) % tiles, grp = (i >> 5) / tiles % groups, k = (i >> 5) / (tiles * groups);
        const int g = lane >> 2, t = lane & 3;
        auto at = [&](int col, int row) { return col < K1 && row < M1 ? W1[(size_t)col * (O * M1) + k * M1 + row] : 0.f; };
        float f[4], d[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            f[e] = at(16 * grp + 4 * t + e, 8 * tile + g);
            d[e] = at(16 * grp + 4 * (g >> 1) + 2 * (e >> 1) + (g & 1), 8 * tile + t + 4 * (e & 1));
        }
        uint32_t hi[4], lo[4];
        const size_t out = (size_t)((i >> 5) * 2) * 32 + lane;
#pragma unroll
        for (int e = 0; e < 4; e++) tf32_split(f[e], hi[e], lo[e]);
        fwd[out] = make_float4(__uint_as_float(hi[0]), __uint_as_float(hi[1]), __uint_as_float(hi[2]), __uint_as_float(hi[3]));
        fwd[out + 32] = make_float4(__uint_as_float(lo[0]), __uint_as_float(lo[1]), __uint_as_float(lo[2]), __uint_as_float(lo[3]));
#pragma unroll
        for (int e = 0; e < 4; e++) tf32_split(d[e], hi[e], lo[e]);
        dxt[out] = make_float4(__uint_as_float(hi[0]), __uint_as_float(hi[1]), __uint_as_float(hi[2]), __uint_as_float(hi[3]));
        dxt[out + 32] = make_float4(__uint_as_float(lo[0]), __uint_as_float(lo[1]), __uint_as_float(lo[2]), __uint_as_float(lo[3]));
    }
}

// Forward.  One CTA per tile of up to 32 positions of one output bucket; its eight warps take the 16-column groups of K1 in
// turn, every lane four 16-byte pieces of x (rows g, g + 8, g + 16, g + 24 of the tile) and the weights' fragments, one group
// ahead of the products.  The warps' sums meet in shared memory; the small layers, the loss, the way back to the first
// layer's pre-activation gradient and the weight gradients of the small layers follow there, one warp per position.
// At 131072 positions (K1 = 2048, M1 = 16) DFWD_BEFORE -> DFWD_AFTER ms against 0.165 for reading x at the copy rate.
// grid = (ntiles, slices of the columns), block = 256, dynamic shared memory = dense_mma_smem<M1>().
template <int M1>
__host__ __device__ constexpr size_t dense_mma_smem() { return (size_t)8 * kDenseTile * M1 * sizeof(float); }

template <int M1>
__global__ void __launch_bounds__(256, (M1 > 16 ? 1 : 2)) dense_forward_mma_kernel(DenseArgs a) {
    step_begin(a.stamp);
    constexpr int NT = mma_tiles<M1>();
    extern __shared__ __align__(16) float dense_smem[];
    __shared__ float s_w2[M1][33], s_b2[32], s_w3[32], s_a1[kDenseTile][M1], loss_part[8];
    __shared__ float s_dz2[kDenseTile][33], s_a2[kDenseTile][33], s_dout[kDenseTile];  // kept per position for the small gradients
    __shared__ int s_pos[kDenseTile];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
    const int2 t = dense_tile_at(a.tiles, blockIdx.x, a.n);
    if (t.y <= 0) return;  // (the launch is sized from the batch size alone)
    if (threadIdx.x < kDenseTile) s_pos[threadIdx.x] = dense_order_at(a.order, t.x + min((int)threadIdx.x, t.y - 1));
    __syncthreads();
    const int k = a.buckets[s_pos[0]];
    const int M2 = a.M[1], OM2 = a.O * M2;
    const int slice = blockIdx.y, slices = gridDim.y;
    // the bucket's small-layer weights: needed only after the long loop
    for (int i = threadIdx.x; i < M1 * M2; i += blockDim.x) s_w2[i / M2][i % M2] = a.W[1][(i / M2) * OM2 + k * M2 + i % M2];
    if (threadIdx.x < 32) {
        const bool on = (int)threadIdx.x < M2;
        s_b2[threadIdx.x] = on ? a.B[1][k * M2 + threadIdx.x] : 0.f;
        s_w3[threadIdx.x] = on && a.n_dense == 3 ? a.W[2][threadIdx.x * a.O + k] : 0.f;
    }
    {
        const int groups = (a.K1 + kMmaCols - 1) / kMmaCols;
        const float* row[4];
#pragma unroll
        for (int r = 0; r < 4; r++) row[r] = a.x + (size_t)s_pos[g + 8 * r] * a.K1 + 4 * t4;
        const float4* table = a.W1f + (size_t)k * groups * NT * 64 + lane;
        float acc[2][NT][4];
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int nt = 0; nt < NT; nt++)
#pragma unroll
                for (int e = 0; e < 4; e++) acc[m][nt][e] = 0.f;
        float4 xv[4], wv[NT][2];
        auto fetch = [&](int grp) {
            const bool in = grp < groups && grp * kMmaCols + 4 * t4 < a.K1;  // K1 is a multiple of four: a piece is inside or outside
#pragma unroll
            for (int r = 0; r < 4; r++) xv[r] = in ? ld_once4(reinterpret_cast<const float4*>(row[r] + grp * kMmaCols)) : make_float4(0, 0, 0, 0);
            if (grp < groups)
#pragma unroll
                for (int nt = 0; nt < NT; nt++)
#pragma unroll
                    for (int part = 0; part < 2; part++) wv[nt][part] = __ldg(table + (size_t)(grp * NT + nt) * 64 + 32 * part);
        };
        fetch(8 * slice + warp);
        for (int grp = 8 * slice + warp; grp < groups; grp += 8 * slices) {
            float xs[4][4];
            uint32_t b[NT][2][4];
#pragma unroll
            for (int r = 0; r < 4; r++) xs[r][0] = xv[r].x, xs[r][1] = xv[r].y, xs[r][2] = xv[r].z, xs[r][3] = xv[r].w;
#pragma unroll
            for (int nt = 0; nt < NT; nt++)
#pragma unroll
                for (int part = 0; part < 2; part++) {
                    b[nt][part][0] = __float_as_uint(wv[nt][part].x), b[nt][part][1] = __float_as_uint(wv[nt][part].y);
                    b[nt][part][2] = __float_as_uint(wv[nt][part].z), b[nt][part][3] = __float_as_uint(wv[nt][part].w);
                }
            fetch(grp + 8 * slices);
            float part_sum[2][NT][4];
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int nt = 0; nt < NT; nt++)
#pragma unroll
                    for (int e = 0; e < 4; e++) part_sum[m][nt][e] = 0.f;
#pragma unroll
            for (int s = 0; s < 2; s++)
#pragma unroll
                for (int m = 0; m < 2; m++) {
                    uint32_t hi[4], lo[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) tf32_split(xs[2 * m + (e & 1)][2 * s + (e >> 1)], hi[e], lo[e]);
#pragma unroll
                    for (int nt = 0; nt < NT; nt++) {
                        mma_tf32(part_sum[m][nt], lo, b[nt][0][2 * s], b[nt][0][2 * s + 1]);
                        mma_tf32(part_sum[m][nt], hi, b[nt][1][2 * s], b[nt][1][2 * s + 1]);
                        mma_tf32(part_sum[m][nt], hi, b[nt][0][2 * s], b[nt][0][2 * s + 1]);
                    }
                }
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int nt = 0; nt < NT; nt++)
#pragma unroll
                    for (int e = 0; e < 4; e++) acc[m][nt][e] += part_sum[m][nt][e];
        }
        float* red = dense_smem + warp * kDenseTile * M1;  // [8][32][M1]
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int nt = 0; nt < NT; nt++)
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int p = 16 * m + g + 8 * (e >> 1), r = 8 * nt + 2 * t4 + (e & 1);
                    if (r < M1) red[p * M1 + r] = acc[m][nt][e];
                }
    }
    const float* red = dense_smem;
    int parts = 8;
    __syncthreads();
    if (slices > 1) {
        // few tiles: the columns are split over CTAs; the one that arrives last adds the slices up, in their order
        __shared__ int last;
        float* mine = a.partial + ((size_t)blockIdx.x * slices + slice) * kDenseTile * M1;
        for (int o = threadIdx.x; o < kDenseTile * M1; o += blockDim.x) {
            float z = 0.f;
#pragma unroll
            for (int w = 0; w < 8; w++) z += red[w * kDenseTile * M1 + o];
            mine[o] = z;
        }
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) last = atomicAdd(a.arrived + blockIdx.x, 1) == slices - 1;
        __syncthreads();
        if (!last) return;
        if (threadIdx.x == 0) a.arrived[blockIdx.x] = 0;
        __threadfence();
        red = a.partial + (size_t)blockIdx.x * slices * kDenseTile * M1;
        parts = slices;
    }
    for (int o = threadIdx.x; o < kDenseTile * M1; o += blockDim.x) {
        float z = 0.f;
#pragma unroll 8
        for (int w = 0; w < parts; w++) z += red[w * kDenseTile * M1 + o];
        const int p = o / M1, r = o % M1;
        const float v = act_fwd(a.act[0], z + a.B[0][k * M1 + r]);
        s_a1[p][r] = v;
        if (a.want_grad && p < t.y) a.a1[(size_t)s_pos[p] * M1 + r] = v;
    }
    __syncthreads();

    float my_loss = 0.f;
    for (int p = warp; p < t.y; p += 8) {  // warp-uniform
        const int b = s_pos[p];
        float z2 = 0.f;
        if (lane < M2) {
#pragma unroll
            for (int c = 0; c < M1; c++) z2 += s_w2[c][lane] * s_a1[p][c];
            z2 += s_b2[lane];
        }
        float o, a2v = 0.f;
        if (a.n_dense == 2) {
            o = __shfl_sync(0xffffffffu, z2, 0);
        } else {
            a2v = lane < M2 ? act_fwd(a.act[1], z2) : 0.f;
            o = warp_sum(s_w3[lane] * a2v) + a.B[2][k];
        }
        if (lane == 0) {
            a.out[b] = o;
            if (a.out_host) a.out_host[b] = o;
        }
        if (!a.want_grad) continue;

        const float s = 1.f / (1.f + expf(-o));
        const float diff = s - a.targets[b];
        my_loss += diff * diff;
        const float dout = (diff + diff) * (s * (1.f - s));
        float dz2;  // gradient at the second layer's pre-activation, lane = row
        if (a.n_dense == 2) {
            dz2 = lane == 0 ? dout : 0.f;
            if (lane == 0 && !a.fuse_small) a.dz[1][b] = dout;
        } else {
            dz2 = lane < M2 ? (s_w3[lane] * dout) * act_bwd(a.act[1], a2v) : 0.f;
            if (!a.fuse_small) {
                if (lane == 0) a.dz[2][b] = dout;
                if (lane < M2) {
                    a.dz[1][(size_t)b * M2 + lane] = dz2;
                    a.a2[(size_t)b * M2 + lane] = a2v;
                }
            }
        }
        s_dz2[p][lane] = dz2;
        s_a2[p][lane] = a2v;
        if (lane == 0) s_dout[p] = dout;
        __syncwarp();
        // dz1[c] = (sum_r2 W2[c][r2] * dz2[r2]) * act'(a1[c]); 32/M1 lanes share one c
        const int c = lane % M1;
        float sum = 0.f;
        for (int r2 = lane / M1; r2 < M2; r2 += 32 / M1) sum += s_w2[c][r2] * s_dz2[p][r2];
#pragma unroll
        for (int o2 = M1; o2 < 32; o2 <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o2);
        if (lane < M1) a.dz[0][(size_t)b * M1 + c] = sum * act_bwd(a.act[0], s_a1[p][c]);
        __syncwarp();
    }
    if (a.want_grad) {
        if (lane == 0) loss_part[warp] = my_loss;
        __syncthreads();
        if (threadIdx.x == 0) {
            float s = 0.f;
            for (int w = 0; w < 8; w++) s += loss_part[w];
            atomicAdd(a.loss, s);
        }
        if (a.fuse_small) {
            // Weight and bias gradients of the narrow layers for this tile's bucket: a thread owns
            // entries (row r, column c) of the M x (K+1) block (column K is the bias), sums over the
            // tile's positions from shared memory and adds the result with one atomic per entry
            // (Matmul::backward on the zero-padded gradient, bias = sum over the batch).
            for (int o = threadIdx.x; o < M2 * (M1 + 1); o += blockDim.x) {  // layer 2: X = a1, dY = dz2
                const int r = o % M2, c = o / M2;
                float sum = 0.f;
                for (int p = 0; p < t.y; p++) sum += s_dz2[p][r] * (c < M1 ? s_a1[p][c] : 1.f);
                if (sum != 0.f) atomicAdd(c < M1 ? a.gW[1] + (size_t)c * OM2 + k * M2 + r : a.gB[1] + k * M2 + r, sum);
            }
            if (a.n_dense == 3)
                for (int o = threadIdx.x; o < M2 + 1; o += blockDim.x) {  // layer 3: X = a2, dY = dout (one row)
                    float sum = 0.f;
                    for (int p = 0; p < t.y; p++) sum += s_dout[p] * (o < M2 ? s_a2[p][o] : 1.f);
                    if (sum != 0.f) atomicAdd(o < M2 ? a.gW[2] + (size_t)o * a.O + k : a.gB[2] + k, sum);
                }
        }
    }
}


// dx[b][c] = sum_r W1[c][k_b][r] * dz1[b][r]   (Matmul::backward, matmul.rs:99-126, on the selected rows).  Same tiles; a
// warp keeps the split gradients of all 32 positions in registers and walks the 16-column groups, storing four neighbouring
// columns per lane and row.  DDX_BEFORE -> DDX_AFTER ms at 131072 positions (0.165 for writing dx at the copy rate).
// grid = ntiles, block = 256.
template <int M1>
__global__ void __launch_bounds__(256, (M1 > 16 ? 1 : 2)) dense_dx_mma_kernel(DenseArgs a, float* dx) {
    step_begin(a.stamp);
    constexpr int NT = mma_tiles<M1>();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
    const int2 t = dense_tile_at(a.tiles, blockIdx.x, a.n);
    if (t.y <= 0) return;
    const int groups = (a.K1 + kMmaCols - 1) / kMmaCols;
    float* row[4];
    uint32_t hi[2][NT][4], lo[2][NT][4];
    int k = 0;
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const int pos = dense_order_at(a.order, t.x + min(g + 8 * r, t.y - 1));
        if (r == 0) k = a.buckets[pos];
        row[r] = dx + (size_t)pos * a.K1 + 4 * t4;
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int rr = 8 * nt + t4 + 4 * i;
                const float v = rr < M1 ? a.dz[0][(size_t)pos * M1 + rr] : 0.f;
                tf32_split(v, hi[r >> 1][nt][(r & 1) + 2 * i], lo[r >> 1][nt][(r & 1) + 2 * i]);
            }
    }
    const float4* table = a.W1d + (size_t)k * groups * NT * 64 + lane;
    float4 wv[NT][2];
    auto fetch = [&](int grp) {
        if (grp < groups)
#pragma unroll
            for (int nt = 0; nt < NT; nt++)
#pragma unroll
                for (int part = 0; part < 2; part++) wv[nt][part] = __ldg(table + (size_t)(grp * NT + nt) * 64 + 32 * part);
    };
    fetch(warp);
    for (int grp = warp; grp < groups; grp += 8) {
        uint32_t b[NT][2][4];
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
#pragma unroll
            for (int part = 0; part < 2; part++) {
                b[nt][part][0] = __float_as_uint(wv[nt][part].x), b[nt][part][1] = __float_as_uint(wv[nt][part].y);
                b[nt][part][2] = __float_as_uint(wv[nt][part].z), b[nt][part][3] = __float_as_uint(wv[nt][part].w);
            }
        fetch(grp + 8);
        const bool in = grp * kMmaCols + 4 * t4 < a.K1;
#pragma unroll
        for (int m = 0; m < 2; m++) {
            float c[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
            for (int nt = 0; nt < NT; nt++)
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    mma_tf32(c[j], lo[m][nt], b[nt][0][2 * j], b[nt][0][2 * j + 1]);
                    mma_tf32(c[j], hi[m][nt], b[nt][1][2 * j], b[nt][1][2 * j + 1]);
                    mma_tf32(c[j], hi[m][nt], b[nt][0][2 * j], b[nt][0][2 * j + 1]);
                }
#pragma unroll
            for (int h = 0; h < 2; h++)
                if (in && 16 * m + 8 * h + g < t.y)
                    *reinterpret_cast<float4*>(row[2 * m + h] + grp * kMmaCols) = make_float4(c[0][2 * h], c[0][2 * h + 1], c[1][2 * h], c[1][2 * h + 1]);
        }
    }
}

// Weight and bias gradient of the first layer: gW[c][k][r] += sum_b [k_b == k] dz1[b][r] * x[b][c].  Positions contract, eight
// a step; r is the M of the product and columns its N: a lane loads four neighbouring columns of two positions, and value j
// of each belongs to column tile j.  A warp owns 64 columns (two groups of 32), a CTA of eight warps 512; the CTA walks a
// run of dense tiles and adds its sums to the gradient when the output bucket changes.  The warp of columns past K1 adds
// the bias gradient.  DWG_BEFORE -> DWG_AFTER ms at 131072 positions (0.165 for reading x at the copy rate).
// grid = (ceil(K1 / 512), runs), block = 256.
constexpr int kWgradCols = 64;
template <int M1>
__global__ void __launch_bounds__(256, (M1 > 16 ? 1 : 2)) dense_wgrad_mma_kernel(DenseArgs a, float* gW, float* gB, int tiles_per_run) {
    step_begin(nullptr);
    constexpr int MT = M1 > 16 ? M1 / 16 : 1;
    __shared__ int s_pos[kDenseTile];
    __shared__ uint32_t s_hi[kDenseTile][M1 + 1], s_lo[kDenseTile][M1 + 1];
    __shared__ float s_dz[kDenseTile][M1 + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
    const int c0 = (blockIdx.x * 8 + warp) * kWgradCols, OM = a.O * M1;
    float acc[MT][8][4];
    float bias_sum = 0.f;
    auto clear = [&]() {
#pragma unroll
        for (int m = 0; m < MT; m++)
#pragma unroll
            for (int j = 0; j < 8; j++)
#pragma unroll
                for (int e = 0; e < 4; e++) acc[m][j][e] = 0.f;
        bias_sum = 0.f;
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
        if (blockIdx.x == 0 && threadIdx.x < M1 && bias_sum != 0.f) atomicAdd(gB + cur * M1 + threadIdx.x, bias_sum);
        clear();
    };
    const int first = blockIdx.y * tiles_per_run, last = min(a.ntiles, first + tiles_per_run);
    for (int tile = first; tile < last; tile++) {
        const int2 t = dense_tile_at(a.tiles, tile, a.n);
        if (t.y <= 0) break;  // (empty tiles come last)
        __syncthreads();
        for (int i = threadIdx.x; i < kDenseTile * M1; i += blockDim.x) {
            const int p = i / M1, r = i % M1, pos = dense_order_at(a.order, t.x + min(p, t.y - 1));
            const float v = p < t.y ? a.dz[0][(size_t)pos * M1 + r] : 0.f;
            tf32_split(v, s_hi[p][r], s_lo[p][r]);
            s_dz[p][r] = v;
            if (r == 0) s_pos[p] = pos;
        }
        __syncthreads();
        const int k = a.buckets[s_pos[0]];
        if (k != cur) {
            flush();
            cur = k;
        }
        if (blockIdx.x == 0 && threadIdx.x < M1)
            for (int p = 0; p < kDenseTile; p++) bias_sum += s_dz[p][threadIdx.x];
        if (c0 >= a.K1) continue;
#pragma unroll
        for (int h = 0; h < 2; h++) {  // the warp's two groups of 32 columns
            const int c = c0 + 32 * h + 4 * g;
            if (c0 + 32 * h >= a.K1) break;
            float4 xv[4][2];
#pragma unroll
            for (int s = 0; s < 4; s++)
#pragma unroll
                for (int i = 0; i < 2; i++)
                    xv[s][i] = c < a.K1 ? ld_once4(reinterpret_cast<const float4*>(a.x + (size_t)s_pos[8 * s + t4 + 4 * i] * a.K1 + c)) : make_float4(0, 0, 0, 0);
            float part_sum[MT][4][4];
#pragma unroll
            for (int m = 0; m < MT; m++)
#pragma unroll
                for (int j = 0; j < 4; j++)
#pragma unroll
                    for (int e = 0; e < 4; e++) part_sum[m][j][e] = 0.f;
#pragma unroll
            for (int s = 0; s < 4; s++) {
                const float v0[4] = {xv[s][0].x, xv[s][0].y, xv[s][0].z, xv[s][0].w}, v1[4] = {xv[s][1].x, xv[s][1].y, xv[s][1].z, xv[s][1].w};
                uint32_t ahi[MT][4], alo[MT][4];
#pragma unroll
                for (int m = 0; m < MT; m++)
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const int r = 16 * m + g + 8 * (e & 1), p = 8 * s + t4 + 4 * (e >> 1);
                        ahi[m][e] = r < M1 ? s_hi[p][r] : 0u;
                        alo[m][e] = r < M1 ? s_lo[p][r] : 0u;
                    }
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    uint32_t h0, l0, h1, l1;
                    tf32_split(v0[j], h0, l0);
                    tf32_split(v1[j], h1, l1);
#pragma unroll
                    for (int m = 0; m < MT; m++) {
                        mma_tf32(part_sum[m][j], ahi[m], l0, l1);
                        mma_tf32(part_sum[m][j], alo[m], h0, h1);
                        mma_tf32(part_sum[m][j], ahi[m], h0, h1);
                    }
                }
            }
#pragma unroll
            for (int m = 0; m < MT; m++)
#pragma unroll
                for (int j = 0; j < 4; j++)
#pragma unroll
                    for (int e = 0; e < 4; e++) acc[m][4 * h + j][e] += part_sum[m][j][e];
        }
    }
    flush();
}

}  // namespace b200
