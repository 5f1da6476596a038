// Networks whose only dense layer is one row per output bucket: forward, loss and the layer's gradients in one pass over x.
//
// Semantics as in kernels_dense.cuh.  A position needs its row of x twice, for the dot product with the bucket's weights and,
// once the loss gradient is known, for the weight gradient; with the row in shared memory it crosses HBM once.  The gradient
// at x is weight times loss gradient, so it is formed where it is used (the feature-transformer backward) and never stored.
//
// A CTA walks a run of units of up to P positions of one output bucket.  Their rows arrive by bulk copies, kOneStages units
// deep, announced by one mbarrier per stage.  Bound by HBM for wide layers (4 K1 bytes per position), by the latency of a
// handful of steps for narrow ones.  us at 16384 positions, against the three kernels it replaces: 45 for 122 at
// K1 = 2048, 21 for 54 at K1 = 256.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "bulk_copy.cuh"
#include "kernels_dense.cuh"

namespace b200 {

constexpr int kOneThreads = 256, kOneStages = 3, kOneMaxK = 4096;

// positions per unit, a power of two: up to 32 KB of rows, so that two CTAs and more share an SM (one waits for its copies
// and look-ups while the other computes) and a batch of a few thousand positions still makes a unit for each
__host__ __device__ inline int one_rows(int K1) {
    int p = 16;
    while (p > 4 && p * K1 > 8192) p >>= 1;
    return p;
}
__host__ __device__ inline size_t one_smem(int K1) { return ((size_t)kOneStages * one_rows(K1) + 1) * K1 * sizeof(float); }

__device__ __forceinline__ float4 square4(float4 v) { return make_float4(v.x * v.x, v.y * v.y, v.z * v.z, v.w * v.w); }

struct OneArgs {
    const float* x;        // [n][K1]
    const int* buckets;    // [n]
    const float* targets;  // [n]
    const int* order;      // as in DenseArgs
    const int2* tiles;
    int n, ntiles, K1, O;
    const float* W;        // [bucket][column]
    const float* B;        // [bucket]
    float* dout;           // [n] loss gradient at the output
    int* kept_bucket;      // [n] the bucket that goes with it
    float* out;            // [n]
    float* out_host;
    float* loss;
    float* gW;             // l1w [column][bucket]
    float* gB;
    int want_grad, units_per_run;
    int* gave_up;          // pinned word, raised if a wait runs out
    unsigned* gmax;        // see FtArgs
    unsigned long long* stamp;
};

// SQUARE: x holds the roots of its values (activation 3 of kernels_ft.cuh).  SCALE: the largest |dout| and |W| are wanted (an
// instantiation of its own: asking at run time costs 1 of 35 us, 16384 positions x 1024 columns, where nobody wants them).
template <bool SQUARE, bool SCALE>
__global__ void __launch_bounds__(kOneThreads) dense_one_kernel(const __grid_constant__ OneArgs a) {
    step_begin(a.stamp);
    extern __shared__ __align__(128) float one_smem_raw[];
    __shared__ uint64_t full[kOneStages];
    __shared__ int s_pos[kOneStages][32], s_rows[kOneStages], s_bucket[kOneStages];
    __shared__ float4 s_sum[kOneThreads];
    __shared__ float s_part[8], s_dout[32], s_loss[32], s_bias;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int P = one_rows(a.K1), per_tile = kDenseTile / P, cols4 = a.K1 / 4;
    float* s_w = one_smem_raw + (size_t)kOneStages * P * a.K1;
    const int total_units = a.ntiles * per_tile, u_begin = blockIdx.x * a.units_per_run, u_end = min(total_units, u_begin + a.units_per_run);
    if (tid == 0) {
        for (int s = 0; s < kOneStages; s++) mbar_init(&full[s], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // Warp 0 fetches: what unit u holds (one unit ahead of its copies, so that the look-ups are not waited for) ...
    int f_pos = 0, f_rows = 0, f_bucket = 0;
    auto look_up = [&](int u) {
        f_rows = 0;
        if (u < u_end) {
            const int2 t = dense_tile_at(a.tiles, u / per_tile, a.n);
            const int at = u % per_tile * P;
            f_rows = max(0, min(P, t.y - at));
            if (lane < f_rows) {
                f_pos = dense_order_at(a.order, t.x + at + lane);
                if (a.O > 1 && lane == 0) f_bucket = a.buckets[f_pos];
            }
        }
    };
    // ... and its rows, one copy per lane
    auto issue = [&](int stage) {
        if (lane < f_rows) s_pos[stage][lane] = f_pos;
        if (lane == 0) {
            s_rows[stage] = f_rows;
            s_bucket[stage] = f_bucket;
            mbar_expect_tx(&full[stage], (uint32_t)f_rows * a.K1 * 4);
        }
        __syncwarp();
        if (lane < f_rows) bulk_load(one_smem_raw + ((size_t)stage * P + lane) * a.K1, a.x + (size_t)f_pos * a.K1, a.K1 * 4, &full[stage]);
    };
    if (warp == 0) {
        look_up(u_begin);
        for (int s = 0; s < kOneStages; s++) {
            issue(s);
            look_up(u_begin + s + 1);
        }
    }
    // the weight gradient: a thread owns up to four float4 of columns; with fewer columns than threads, `groups` threads share
    // a column piece and split the rows
    const int width = min(kOneThreads, cols4), groups = kOneThreads / width, col = tid % width, group = tid / width;
    float4 acc[4];
    float g_bias = 0.f, my_loss = 0.f;
    unsigned largest_dout = 0, largest_w = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) acc[i] = make_float4(0, 0, 0, 0);
    int cur = -1;
    auto flush = [&]() {
        if (cur < 0 || !a.want_grad) return;  // (uniform)
        if (groups > 1) {  // (then a thread owns one piece) the threads of a column piece add up first
            __syncthreads();
            if (group < groups && group > 0) s_sum[(group - 1) * width + col] = acc[0];
            __syncthreads();
            if (group == 0)
                for (int o = 0; o < groups - 1; o++) acc[0] = add4(acc[0], s_sum[o * width + col]);
        }
        if (group == 0)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int c4 = col + i * kOneThreads;
                if (c4 >= cols4) break;
                float* g = a.gW + (size_t)4 * c4 * a.O + cur;
                if (a.O == 1) {
                    atomicAdd(reinterpret_cast<float4*>(g), acc[i]);
                } else {
                    atomicAdd(g, acc[i].x), atomicAdd(g + a.O, acc[i].y), atomicAdd(g + 2 * a.O, acc[i].z), atomicAdd(g + 3 * a.O, acc[i].w);
                }
            }
#pragma unroll
        for (int i = 0; i < 4; i++) acc[i] = make_float4(0, 0, 0, 0);
        if (warp == 0) {  // (one addition per CTA: the sum of many rounds once for each)
            const float sum = warp_sum(g_bias);
            if (lane == 0 && sum != 0.f) atomicAdd(a.gB + cur, sum);
        }
        g_bias = 0.f;
    };
    __syncthreads();
    const int per_row = kOneThreads / P, row = tid / per_row, in_row = tid % per_row;  // the dot products: threads per row
    for (int u = u_begin; u < u_end; u++) {
        const int step = u - u_begin, stage = step % kOneStages;
        const int rows = s_rows[stage], k = s_bucket[stage];
        if (rows > 0) {
            if (k != cur) {  // (uniform) the bucket's weights
                flush();
                cur = k;
                if (tid == 0) s_bias = __ldg(a.B + k);
                for (int c = tid; c < cols4; c += kOneThreads) {
                    const float4 w = __ldg(reinterpret_cast<const float4*>(a.W + (size_t)k * a.K1) + c);
                    reinterpret_cast<float4*>(s_w)[c] = w;
                    if (SCALE) largest_w = max(max(largest_w, max(magnitude(w.x), magnitude(w.y))), max(magnitude(w.z), magnitude(w.w)));
                }
                __syncthreads();
            }
            const float target = a.want_grad && in_row == 0 && row < rows ? __ldg(a.targets + s_pos[stage][row]) : 0.f;  // (arrives under the sums)
            if (!mbar_wait(&full[stage], (step / kOneStages) & 1)) {
                *a.gave_up = 1;
                return;
            }
            const float4* x = reinterpret_cast<const float4*>(one_smem_raw + (size_t)stage * P * a.K1);
            float dot = 0.f;
            if (row < rows) {
                const float4* xr = x + (size_t)row * cols4;
                float4 d4 = make_float4(0, 0, 0, 0);
#pragma unroll 4
                for (int c = in_row; c < cols4; c += per_row) {
                    float4 v = xr[c];
                    const float4 w = reinterpret_cast<const float4*>(s_w)[c];
                    if (SQUARE) v = square4(v);
                    d4.x += v.x * w.x, d4.y += v.y * w.y, d4.z += v.z * w.z, d4.w += v.w * w.w;
                }
                dot = (d4.x + d4.y) + (d4.z + d4.w);
            }
            for (int o = min(16, per_row / 2); o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
            if (per_row > 32) {  // two warps share a row
                if (lane == 0) s_part[warp] = dot;
                __syncthreads();
                dot = s_part[warp & ~1] + s_part[warp | 1];
            }
            if (in_row == 0) {
                float dout = 0.f;
                if (row < rows) {
                    const int b = s_pos[stage][row];
                    const float o = dot + s_bias;
                    a.out[b] = o;
                    if (a.out_host) a.out_host[b] = o;
                    if (a.want_grad) {
                        const float s = 1.f / (1.f + expf(-o));
                        const float diff = s - target;
                        s_loss[row] = diff * diff;
                        dout = (diff + diff) * (s * (1.f - s));
                        a.dout[b] = dout;
                        a.kept_bucket[b] = k;
                        if (SCALE) largest_dout = max(largest_dout, magnitude(dout));
                    }
                }
                s_dout[row] = dout;
            }
            __syncthreads();
            if (a.want_grad) {
                if (tid < rows) g_bias += s_dout[tid], my_loss += s_loss[tid];
                if (group < groups)
                    for (int r = group; r < rows; r += groups) {
                        const float d = s_dout[r];
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const int c4 = col + i * kOneThreads;
                            if (c4 >= cols4) break;
                            float4 v = x[(size_t)r * cols4 + c4];
                            if (SQUARE) v = square4(v);
                            acc[i].x += d * v.x, acc[i].y += d * v.y, acc[i].z += d * v.z, acc[i].w += d * v.w;
                        }
                    }
            }
        } else if (!mbar_wait(&full[stage], (step / kOneStages) & 1)) {
            *a.gave_up = 1;
            return;
        }
        __syncthreads();  // the stage is free again (and its new description is read several barriers later)
        if (warp == 0 && u + kOneStages < u_end) {
            issue(stage);
            look_up(u + kOneStages + 1);
        }
    }
    flush();
    if (a.want_grad) {
        __shared__ unsigned s_largest[2][kOneThreads / 32];
        if (SCALE) {
            largest_dout = __reduce_max_sync(0xffffffffu, largest_dout);
            largest_w = __reduce_max_sync(0xffffffffu, largest_w);
            if (lane == 0) s_largest[0][warp] = largest_dout, s_largest[1][warp] = largest_w;
        }
        if (tid < 32) s_loss[tid] = tid < P ? my_loss : 0.f;
        __syncthreads();
        if (SCALE && (warp == 1 || warp == 2)) raise_magnitude(a.gmax + warp - 1, s_largest[warp - 1][lane % (kOneThreads / 32)]);
        if (warp == 0) {
            const float sum = warp_sum(s_loss[lane]);
            if (lane == 0 && sum != 0.f) atomicAdd(a.loss, sum);
        }
    }
}

// The gradient at x of such a network, for inspection: dx[b][c] = W[bucket of b][c] * dout[b].
static __global__ void dense_one_dx_kernel(const float* W, const float* dout, const int* kept_bucket, float* dx, int n, int K1) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < (size_t)n * K1; i += (size_t)gridDim.x * blockDim.x) {
        const int b = (int)(i / K1), c = (int)(i % K1);
        dx[i] = W[(size_t)kept_bucket[b] * K1 + c] * dout[b];
    }
}

}  // namespace b200
