// Output-bucketed dense layers, sigmoid-MSE loss and their backward.
//
// Reference semantics (jw1912/bullet): every dense layer is `W.matmul(x) + b`
// (crates/compiler/src/model/builder.rs:145-147, Matmul::evaluate in
// crates/compiler/src/tensor/operation/linear/matmul.rs:62-93) computed for ALL output
// buckets and then narrowed by `select` (crates/compiler/src/tensor/operation/index/select.rs:12-26);
// its backward pads the selected gradient with zeros (select.rs:93-110).  Here only the
// selected bucket's rows are ever computed, which gives the same numbers: the rows of the
// other buckets contribute exactly zero to every gradient.
// Weights are column-major: element (bucket k, row r, column c) of layer i sits at
// W[c * (O*M_i) + k*M_i + r].
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels_group.cuh"

namespace b200 {

constexpr int kDenseWarpPos = 4;  // positions of a tile (kDenseTile of them, 8 warps) that each warp takes
constexpr int kDenseChunk = 128;  // first-layer columns staged in shared memory per round

struct DenseArgs {
    const float* x;        // [n][K1] dense-stack input
    const int* buckets;    // [n] output bucket per position
    const float* targets;  // [n]
    const int* order;      // [n] position ids grouped by output bucket, or null (one bucket): as they come
    const int2* tiles;     // [ntiles] (begin, count <= kDenseTile) ranges of `order`, one bucket each, or null as well
    int n, ntiles, K1, O, n_dense;
    int M[3], act[3];
    const float* W[3];
    const float* B[3];
    const float* W1g;  // first-layer weights regrouped as [bucket][column][row] (fewer than four rows)
    const uint32_t* W1f; // ... or as the fragment tables of kernels_dense_mma.cuh
    const uint32_t* W1d;
    float* partial;    // [part][tile][32][M1] sums of slices of the first layer's columns
    uint32_t* dz_frag; // dz[0] as the tensor pipe's operand of the weight gradient (dense_small_mma_kernel)
    float* a1;         // [n][M1] activated layer-1 output (kept for the weight gradients)
    float* a2;         // [n][M2]
    float* dz[3];      // gradient at each layer's selected pre-activation: [n][M_i]
    float* out;        // [n] network output
    float* out_host;   // the same in pinned host memory, or null
    float* loss;       // scalar, accumulated
    int want_grad;
    unsigned long long* stamp;  // as in FtArgs
    int* gave_up;               // pinned word, raised if a wait for copies runs out
    unsigned* gmax;             // see FtArgs
    // gradient tensors (of the kernels that form them on the way)
    float* gW[3];
    float* gB[3];
};

// tile `i` of a batch of n positions, and the position at place `at` of the order
__device__ __forceinline__ int2 dense_tile_at(const int2* tiles, int i, int n) {
    return tiles ? tiles[i] : make_int2(i * kDenseTile, min(kDenseTile, n - i * kDenseTile));
}
__device__ __forceinline__ int dense_order_at(const int* order, int at) { return order ? order[at] : at; }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ float act_fwd(int act, float v) { return act == 0 ? v : ft_act_fwd(act, v); }
__device__ __forceinline__ float act_bwd(int act, float y) { return act == 0 ? 1.f : ft_act_bwd(act, y); }

// Network outputs into pinned host memory, coalesced (they are computed in the order of the output buckets).
static __global__ void __launch_bounds__(256) copy_outputs_kernel(const float* out, float* host, int n) {
    step_begin(nullptr);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) host[i] = out[i];
}

// l1w is stored column-major over ALL buckets' rows, so the M1 rows of one bucket for
// consecutive columns lie O*M1 floats apart.  The kernels below read the regrouped copy
// W1g[bucket][column][row], in which one bucket's weights for a run of columns are contiguous.
__global__ void dense_regroup_kernel(const float* __restrict__ W1, float* __restrict__ W1g, int K1, int O, int M1) {
    const int total = K1 * O * M1;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const int r = i % M1, c = (i / M1) % K1, k = i / (M1 * K1);
        W1g[i] = W1[(size_t)c * (O * M1) + k * M1 + r];
    }
}

__device__ __forceinline__ void dense_cp_async16(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void dense_cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void dense_cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Stages columns [chunk*128, chunk*128+128) of bucket k's first-layer weights; columns past
// K1 are zero-filled.  All 256 threads take part.
template <int M1>
__device__ __forceinline__ void dense_stage_chunk(const DenseArgs& a, int k, int chunk, float* buf) {
    const int c_begin = chunk * kDenseChunk;
    const float* src = a.W1g + ((size_t)k * a.K1 + c_begin) * M1;
    for (int i = threadIdx.x; i < kDenseChunk * M1; i += blockDim.x) buf[i] = c_begin + i / M1 < a.K1 ? __ldg(src + i) : 0.f;
}

template <int M1>
__device__ __forceinline__ void dense_read_weights(const float* buf, int c, float (&w)[M1]) {
#pragma unroll
    for (int r = 0; r < M1; r++) w[r] = buf[c * M1 + r];
}

// One CTA per tile of up to 32 positions of the same output bucket, four per warp.  The
// bucket's first-layer weights AND the tile's rows of x stream through shared memory in
// 128-column chunks, three chunks in flight (cp.async), so no global latency sits between
// the chunks; lane l takes columns l, l+32, l+64, l+96 of a chunk.  After the K1-long dot
// products the tiny remaining layers, the loss and the backward pass down to the first
// layer's pre-activation gradient follow per position.  grid = ntiles, block = 256, dynamic
// shared memory = dense_fwd_smem<M1>().
constexpr int kDenseStages = 3;
template <int M1>
__host__ __device__ constexpr size_t dense_fwd_smem() {
    return (size_t)kDenseStages * (kDenseChunk * M1 + kDenseTile * kDenseChunk) * sizeof(float);
}

template <int M1>
__global__ void __launch_bounds__(256, 2) dense_forward_kernel(DenseArgs a) {
    step_begin(a.stamp);
    constexpr int P = kDenseWarpPos;
    constexpr int kStageFloats = kDenseChunk * M1 + kDenseTile * kDenseChunk;
    extern __shared__ __align__(16) float dense_smem[];
    __shared__ float loss_part[8];
    __shared__ int s_pos[kDenseTile];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int2 t = dense_tile_at(a.tiles, blockIdx.x, a.n);
    if (t.y <= 0) return;  // (the launch is sized from the batch size alone)
    if (threadIdx.x < kDenseTile) s_pos[threadIdx.x] = dense_order_at(a.order, t.x + min((int)threadIdx.x, t.y - 1));
    __syncthreads();
    const int k = a.buckets[s_pos[0]];
    const int npos = max(0, min(P, t.y - warp * P));
    int pos[P];
#pragma unroll
    for (int j = 0; j < P; j++) pos[j] = s_pos[min(warp * P + j, t.y - 1)];
    float acc[P][M1];
#pragma unroll
    for (int j = 0; j < P; j++)
#pragma unroll
        for (int r = 0; r < M1; r++) acc[j][r] = 0.f;
    const int nchunks = (a.K1 + kDenseChunk - 1) / kDenseChunk;
    // one cp.async group per chunk: the bucket's weights and the tile's x for 128 columns
    auto stage = [&](int ch) {
        if (ch < nchunks) {
            float* wb = dense_smem + (ch % kDenseStages) * kStageFloats;
            float* xb = wb + kDenseChunk * M1;
            dense_stage_chunk<M1>(a, k, ch, wb);
            for (int i = threadIdx.x; i < kDenseTile * (kDenseChunk / 4); i += blockDim.x) {
                const int p = i / (kDenseChunk / 4), q = i % (kDenseChunk / 4);
                const int c = ch * kDenseChunk + q * 4;  // K1 is a multiple of four: a quad is inside or outside
                float* dst = xb + p * kDenseChunk + q * 4;
                if (c < a.K1)
                    dense_cp_async16(dst, a.x + (size_t)s_pos[p] * a.K1 + c);
                else
                    *reinterpret_cast<float4*>(dst) = make_float4(0, 0, 0, 0);
            }
        }
        dense_cp_commit();  // an empty group past the end keeps the group count in step with `ch`
    };
    stage(0);
    stage(1);
    for (int ch = 0; ch < nchunks; ch++) {
        stage(ch + 2);
        dense_cp_wait<kDenseStages - 1>();  // chunk ch has landed
        __syncthreads();
        if (npos) {
            const float* wb = dense_smem + (ch % kDenseStages) * kStageFloats;
            const float* xb = wb + kDenseChunk * M1 + (warp * P) * kDenseChunk;
#pragma unroll
            for (int jj = 0; jj < 4; jj++) {
                float w[M1];
                dense_read_weights<M1>(wb, jj * 32 + lane, w);
#pragma unroll
                for (int j = 0; j < P; j++) {
                    const float xv = xb[j * kDenseChunk + jj * 32 + lane];
#pragma unroll
                    for (int r = 0; r < M1; r++) acc[j][r] += w[r] * xv;
                }
            }
        }
        __syncthreads();  // the stage read here is refilled by the next iteration
    }
    float my_loss = 0.f;
#pragma unroll
    for (int j = 0; j < P; j++) {
        if (j >= npos) break;  // warp-uniform
        const int b = pos[j];
        float a1v[M1];
#pragma unroll
        for (int r = 0; r < M1; r++) a1v[r] = act_fwd(a.act[0], warp_sum(acc[j][r]) + a.B[0][k * M1 + r]);

        float o;        // network output
        float a2v = 0;  // lane r2 holds a2[r2] when there are three layers
        if (a.n_dense == 1) {
            o = a1v[0];
        } else {
            const int M2 = a.M[1], OM2 = a.O * M2;
            float z2 = 0.f;
            if (lane < M2) {
#pragma unroll
                for (int c = 0; c < M1; c++) z2 += a.W[1][c * OM2 + k * M2 + lane] * a1v[c];
                z2 += a.B[1][k * M2 + lane];
            }
            if (a.n_dense == 2) {
                o = __shfl_sync(0xffffffffu, z2, 0);
            } else {
                a2v = lane < M2 ? act_fwd(a.act[1], z2) : 0.f;
                const float term = lane < M2 ? a.W[2][lane * a.O + k] * a2v : 0.f;
                o = warp_sum(term) + a.B[2][k];
            }
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
        float dz1[M1];
        if (a.n_dense == 1) {
            dz1[0] = dout;  // M1 == 1, no activation on the last layer
        } else if (a.n_dense == 2) {
            if (lane == 0) a.dz[1][b] = dout;
#pragma unroll
            for (int c = 0; c < M1; c++) dz1[c] = (a.W[1][c * a.O + k] * dout) * act_bwd(a.act[0], a1v[c]);
        } else {
            const int M2 = a.M[1], OM2 = a.O * M2;
            if (lane == 0) a.dz[2][b] = dout;
            float dz2 = 0.f;
            if (lane < M2) {
                dz2 = (a.W[2][lane * a.O + k] * dout) * act_bwd(a.act[1], a2v);
                a.dz[1][(size_t)b * M2 + lane] = dz2;
                a.a2[(size_t)b * M2 + lane] = a2v;
            }
#pragma unroll
            for (int c = 0; c < M1; c++) {
                const float term = lane < M2 ? a.W[1][c * OM2 + k * M2 + lane] * dz2 : 0.f;
                dz1[c] = warp_sum(term) * act_bwd(a.act[0], a1v[c]);
            }
        }
#pragma unroll
        for (int c = 0; c < M1; c++)
            if (lane == (c & 31)) {
                a.dz[0][(size_t)b * M1 + c] = dz1[c];
                if (a.n_dense > 1) a.a1[(size_t)b * M1 + c] = a1v[c];
            }
    }
    if (a.want_grad) {
        if (lane == 0) loss_part[warp] = my_loss;
        __syncthreads();
        if (threadIdx.x == 0) {
            float s = 0.f;
            for (int w = 0; w < 8; w++) s += loss_part[w];
            atomicAdd(a.loss, s);
        }
    }
}

// dx[b][c] = sum_r W1[c][k_b][r] * dz1[b][r]   (Matmul::backward, matmul.rs:99-126, on the
// selected rows).  Same tiling and weight staging as the forward; grid = ntiles, block = 256.
template <int M1>
__global__ void __launch_bounds__(256, 2) dense_dx_kernel(DenseArgs a, float* dx) {
    step_begin(a.stamp);
    constexpr int P = kDenseWarpPos;
    __shared__ __align__(16) float wbuf[2][kDenseChunk * M1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int2 t = dense_tile_at(a.tiles, blockIdx.x, a.n);
    if (t.y <= 0) return;
    const int k = a.buckets[dense_order_at(a.order, t.x)];
    const int npos = max(0, min(P, t.y - warp * P));
    int pos[P];
#pragma unroll
    for (int j = 0; j < P; j++) pos[j] = dense_order_at(a.order, npos ? t.x + warp * P + min(j, npos - 1) : t.x);
    float g[P][M1];
#pragma unroll
    for (int j = 0; j < P; j++)
#pragma unroll
        for (int r = 0; r < M1; r++) g[j][r] = a.dz[0][(size_t)pos[j] * M1 + r];
    const int nchunks = (a.K1 + kDenseChunk - 1) / kDenseChunk;
    unsigned largest = 0;
    dense_stage_chunk<M1>(a, k, 0, wbuf[0]);
    for (int ch = 0; ch < nchunks; ch++) {
        if (ch + 1 < nchunks) dense_stage_chunk<M1>(a, k, ch + 1, wbuf[(ch + 1) & 1]);
        __syncthreads();
        if (npos) {
            const float* buf = wbuf[ch & 1];
#pragma unroll
            for (int jj = 0; jj < 4; jj++) {
                const int c = ch * kDenseChunk + jj * 32 + lane;
                float w[M1];
                dense_read_weights<M1>(buf, jj * 32 + lane, w);
#pragma unroll
                for (int j = 0; j < P; j++) {
                    float s = 0.f;
#pragma unroll
                    for (int r = 0; r < M1; r++) s += w[r] * g[j][r];
                    if (j < npos && c < a.K1) {
                        dx[(size_t)pos[j] * a.K1 + c] = s;
                        largest = max(largest, magnitude(s));
                    }
                }
            }
        }
        __syncthreads();
    }
    raise_magnitude(a.gmax, largest);
}

// Weight and bias gradient of one dense layer: gW[c][k][r] += sum_b [k_b == k] dY[b][r] * X[b][c],
// gB[k][r] += sum_b [k_b == k] dY[b][r]  (Matmul::backward on the zero-padded gradient,
// reduce over the batch for the bias: model/builder.rs:263-267).
// Positions are visited in bucket-sorted order (`order`), so a thread keeps M running sums
// for the current bucket and flushes them with atomics only when the bucket changes.
// A thread owns four neighbouring columns (16 bytes of x per position, prefetched eight positions
// ahead through shared memory); the thread after the last column owns the bias.  grid = (ceil((K/4 + 1) / 128), chunks), block = 128.
struct WgradArgs {
    const float* X;      // [n][K]
    const float* dY;     // [n][M]
    const int* order;    // [n] position ids sorted by bucket, or null = identity
    const int* buckets;  // [n] by position id
    int n, K, O, chunk_len;
    float* gW;
    float* gB;
};

template <int M>
__global__ void __launch_bounds__(128) dense_wgrad_kernel(WgradArgs a) {
    step_begin(nullptr);
    constexpr int S = 64;  // positions staged per round
    __shared__ int s_pos[S], s_bucket[S];
    __shared__ __align__(16) float s_dy[S][M];
    const int c = 4 * (blockIdx.x * blockDim.x + threadIdx.x);  // this thread's four columns c .. c+3
    const bool is_col = c < a.K, is_bias = c == a.K;             // K is a multiple of four
    const int OM = a.O * M;
    const int begin = blockIdx.y * a.chunk_len, end = min(a.n, begin + a.chunk_len);
    float acc[4][M];
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
        for (int r = 0; r < M; r++) acc[q][r] = 0.f;
    int cur = -1;
    auto flush = [&]() {  // one column's M rows are contiguous: 128-bit reductions when M allows
        if (cur >= 0 && (is_col || is_bias)) {
#pragma unroll
            for (int q = 0; q < 4; q++) {
                float* dst = is_col ? a.gW + (size_t)(c + q) * OM + cur * M : a.gB + cur * M;
                if (is_col || q == 0) {
                    if (M % 4 == 0) {
#pragma unroll
                        for (int r = 0; r < M; r += 4)
                            atomicAdd(reinterpret_cast<float4*>(dst + r), make_float4(acc[q][r], acc[q][r + 1], acc[q][r + 2], acc[q][r + 3]));
                    } else {
#pragma unroll
                        for (int r = 0; r < M; r++)
                            if (acc[q][r] != 0.f) atomicAdd(dst + r, acc[q][r]);
                    }
                }
#pragma unroll
                for (int r = 0; r < M; r++) acc[q][r] = 0.f;
            }
        }
    };
    // x reaches the thread through a private ring of D shared-memory slots filled by cp.async:
    // D positions' loads stay in flight at no register cost, so HBM latency hides behind the FMAs
    constexpr int D = 8;
    __shared__ float4 s_x[D][128];
    float4* my_slot = &s_x[0][threadIdx.x];
    for (int base = begin; base < end; base += S) {
        const int cnt = min(S, end - base);
        __syncthreads();
        for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
            const int pos = a.order ? a.order[base + i] : base + i;
            s_pos[i] = pos;
            s_bucket[i] = a.buckets[pos];
        }
        __syncthreads();
        for (int i = threadIdx.x; i < cnt * M; i += blockDim.x) s_dy[i / M][i % M] = a.dY[(size_t)s_pos[i / M] * M + i % M];
#pragma unroll
        for (int u = 0; u < D; u++) {
            if (u < cnt && is_col) dense_cp_async16(my_slot + u * 128, a.X + (size_t)s_pos[u] * a.K + c);
            dense_cp_commit();
        }
        __syncthreads();
        for (int j = 0; j < cnt; j++) {
            dense_cp_wait<D - 1>();  // position j's 16 bytes have landed
            const float4 xv = is_col ? my_slot[(j & (D - 1)) * 128] : make_float4(is_bias ? 1.f : 0.f, 0.f, 0.f, 0.f);  // the bias "column" sees x = 1
            const int k = s_bucket[j];
            if (k != cur) {
                flush();
                cur = k;
            }
            const float xs[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
            for (int r = 0; r < M; r++) {
                const float dy = s_dy[j][r];
#pragma unroll
                for (int q = 0; q < 4; q++) acc[q][r] += dy * xs[q];
            }
            // refill the slot just read (after its value has been used) with position j + D
            if (j + D < cnt && is_col) dense_cp_async16(my_slot + (j & (D - 1)) * 128, a.X + (size_t)s_pos[j + D] * a.K + c);
            dense_cp_commit();
        }
    }
    flush();
}

// Weight and bias gradients of the narrow layers after the first, all in one launch: one CTA
// per tile of up to 32 positions of one output bucket (the tiles of the forward).  For layer
// l >= 1 with input X = the activated output of layer l-1 (K values per position) and dY = the
// gradient at its selected pre-activation (M values): a thread owns entries (row r, column c)
// of the bucket's M x (K+1) block (column K is the bias), sums dY[p][r] * X[p][c] over the
// tile's positions from shared memory and adds the result with one atomic per entry.
// grid = ntiles, block = 256.
struct SmallGradArgs {
    const int* order;
    const int2* tiles;
    const int* buckets;
    int n, O, n_layers;  // layers handled here: dense layers 1 .. n_dense-1
    int K[2], M[2];
    const float* X[2];   // [n][K]
    const float* dY[2];  // [n][M]
    float* gW[2];
    float* gB[2];
};

static __global__ void __launch_bounds__(256) dense_small_grads_kernel(SmallGradArgs a) {
    step_begin(nullptr);
    __shared__ float s_x[32][33], s_dy[32][33];
    __shared__ int s_pos[32];
    const int2 t = dense_tile_at(a.tiles, blockIdx.x, a.n);
    if (t.y <= 0) return;
    if (threadIdx.x < t.y) s_pos[threadIdx.x] = dense_order_at(a.order, t.x + threadIdx.x);
    __syncthreads();
    const int k = a.buckets[s_pos[0]];
    for (int l = 0; l < a.n_layers; l++) {
        const int K = a.K[l], M = a.M[l], OM = a.O * M;
        __syncthreads();
        for (int i = threadIdx.x; i < t.y * (K + 1); i += blockDim.x) {
            const int p = i / (K + 1), c = i % (K + 1);
            s_x[p][c] = c < K ? a.X[l][(size_t)s_pos[p] * K + c] : 1.f;
        }
        for (int i = threadIdx.x; i < t.y * M; i += blockDim.x) {
            const int p = i / M, r = i % M;
            s_dy[p][r] = a.dY[l][(size_t)s_pos[p] * M + r];
        }
        __syncthreads();
        for (int o = threadIdx.x; o < M * (K + 1); o += blockDim.x) {
            const int r = o % M, c = o / M;
            float sum = 0.f;
            for (int p = 0; p < t.y; p++) sum += s_dy[p][r] * s_x[p][c];
            if (sum != 0.f) atomicAdd(c < K ? a.gW[l] + (size_t)c * OM + k * M + r : a.gB[l] + k * M + r, sum);
        }
    }
}

}  // namespace b200
