// Feature-transformer kernels: the sparse affine layer on both perspectives with the
// bias, activation, pairwise product and stm|nstm concat fused in, and its backward.
//
// Reference semantics (jw1912/bullet): SparseMatmul::evaluate
// (crates/compiler/src/tensor/operation/linear/sparse.rs:86-119) sums table rows in
// slot order starting from 0 and skips invalid slots; the bias is added afterwards
// (crates/compiler/src/model/builder.rs:145-147); activations and their
// derivatives-from-output follow crates/compiler/src/tensor/operation/autograd/dfo.rs:47-119;
// the backward adds the incoming gradient to one table row per valid slot
// (sparse.rs:151-187).  Both forward kernels add rows in slot order, so their
// pre-activations are bit-identical to the interpreter's fp32 result.
//
// Two families (the backward of tables of few rows has a third form, kernels_ft_mma.cuh):
//   *_gather : one warp per (position, perspective, chunk of columns); rows come
//              straight from the table (L2/HBM), gradients go out as 128-bit
//              global reductions.  Works for any index set.
//   *_tiled  : for inputs whose active features of one perspective all lie in one
//              aligned block of R table rows (king buckets).  A forward CTA stages one
//              R x 64-column tile of the table in shared memory and serves every
//              (position, perspective) of that block from it; a backward CTA
//              stages the gradients of a run of them and sums these row by row from lists.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "launch.cuh"
#include "peer_flags.cuh"
#include "tmem.cuh"

namespace b200 {

constexpr uint32_t kNoFeature = 0xFFFFu;
constexpr int kStatusOutsideBlock = 1;  // a feature fell outside its position's declared row block

// A kernel's largest dynamic shared memory holds for the process, whatever network asks: always all there is.
template <class K>
cudaError_t allow_smem(K* kernel) {
    cudaFuncAttributes attr;
    const cudaError_t e = cudaFuncGetAttributes(&attr, reinterpret_cast<const void*>(kernel));
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(227 * 1024 - attr.sharedSizeBytes));
}

struct FtArgs {
    const float* table;   // [n_inputs][H] effective weights: l0w, or l0w + tiled l0f already merged
    const float* factor;  // forward only: [factor_rows][H] l0f to be added to `table` (= l0w) on the fly, or null
    int factor_rows;
    int block_rows;       // gather forward only: > 0 drops features outside the block of their pair's first one, as the tiled kernels do
    const float* bias;    // [H]
    const uint16_t* idx_stm;
    const uint16_t* idx_nstm;  // [n][nnz] each, 0xFFFF = empty slot
    int n, nnz, H, n_inputs, act;
    float* x;         // dense-stack input: [n][2H], or [n][H] with pairwise
    float* u;         // pairwise only: crelu outputs [n][2][H]
    const float* dx;  // backward: gradient at x, or (null) what it is the product of, for networks whose only dense layer is
    const float* w1;          // one row per output bucket: the layer's weights [bucket][K1],
    const float* dout;        // [n] the loss gradient at the output
    const int* out_bucket;    // [n] and the bucket
    float* g_table;   // backward: [n_inputs][H] gradient of the table
    float* g_bias;    // backward: [H]
    unsigned long long* stamp;  // of a step that keeps its own time: where the kernel's start goes
    unsigned long long* stamp_end;  // forward: the step's last stamp, cleared
    float4* zero;     // forward: the gradient buffer, where this kernel clears it (zero4 float4s), or null
    long long zero4;
    unsigned* gmax;   // the largest |dx| (or |dout|, and |w1| behind it) of the step, as bits: the forward clears them, the dense
                      // kernels raise them, ft_backward_mma_kernel scales by them
    int* gave_up;     // pinned word, raised if a wait inside a kernel runs out
    int* status;      // gather forward only: where a feature outside its pair's block is reported, or null
};

__device__ __forceinline__ void ft_step_begin(const FtArgs& a) {
    step_begin(a.stamp);
    if (a.stamp_end && threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0) *a.stamp_end = 0;
    if (a.gmax && threadIdx.x < 2 && blockIdx.x == 0 && blockIdx.y == 0) a.gmax[threadIdx.x] = 0u;
    if (a.zero) {  // nothing adds to it before the kernels that follow
        const long long per = (long long)gridDim.x * gridDim.y * blockDim.x;
        for (long long i = ((long long)blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x; i < a.zero4; i += per) a.zero[i] = make_float4(0, 0, 0, 0);
    }
}

struct TileArgs {
    int block_rows;          // R
    int nslabs;              // column slabs of 64 (the last may be partly filled)
    // A launch covers the row blocks [first_block, last_block) with gridDim.x CTAs.  The work of those
    // blocks is laid out in one line (block by block; inside a block column slab by column slab; inside a
    // slab pair by pair, for the backward chunk by chunk) and CTA k takes the k-th of gridDim.x near-equal
    // contiguous pieces of that line: every SM gets the same amount of work whatever the blocks hold, and
    // a tile is loaded about once per (block, slab) and SM that touches it.
    int first_block, last_block;
    const int2* pairs;       // [2n] (pair id = position*2 + perspective, number of active rows) grouped by block
    const int* block_begin;  // [nblocks+1] offsets into pairs
    const int* chunk_begin;  // backward: [nblocks+1] first chunk of every block
    int* status;
    // written by the grouping (kernels_group.cuh): for the i-th pair in visiting
    // order its active rows (local to the pair's block) in slot order; the tail of the last
    // 16-byte group is filled with the index of the all-zero row (= block_rows) and never walked
    const uint16_t* lists;  // [2n][list_len]
    int list_len;     // nnz rounded up to a multiple of 8 (16-byte groups)
    int walk_warps;   // forward: see ft_fwd_warps
    int fill_steps;   // forward: rounds of 128 rows of a tile
    // backward only: the visiting order cut into chunks of at most kChunkMost pairs that never
    // straddle a block, and per chunk the row-major lists built by ft_csr_kernel
    const int4* chunks;            // [nchunks] (block, first index into `pairs`, pairs, 0)
    uint16_t* csr_ent;             // [nchunks][ent_cap] pairs of the chunk grouped by row, every list starting on 8 bytes
    int* csr_start;                // [nchunks][start_cap] entries, pieces, two unused words, then the pieces (see ft_bwd_start_cap)
    int ent_cap, start_cap;
    int chunk_len;  // CP: most pairs per chunk
    int wide;       // 1024 threads per CTA, one per SM; else 512 and two
    // backward only, data-parallel runs: the last CTA of every row block tells all ranks that the block's
    // gradient is complete (done_count null: nobody is told)
    BucketSignal sig;
};

__device__ __forceinline__ float crelu_f(float v) { return fminf(fmaxf(v, 0.f), 1.f); }

// activation of the FT output: 1 = crelu, 2 = screlu, 3 = screlu kept as its root: the buffer holds the clamped value, and
// whoever reads it squares it.  The root of fl(c * c) is c to the last bit, so the derivative needs no square root (which made
// the backward's staging twice as long as with crelu) and nothing else changes.
__device__ __forceinline__ float ft_act_fwd(int act, float v) {
    const float c = crelu_f(v);
    return act == 2 ? c * c : c;
}
// d(activation)/d(input) as a function of the activation OUTPUT y (dfo.rs:70-88)
__device__ __forceinline__ float ft_act_bwd(int act, float y) {
    if (act == 3) {
        const float sq = __fmul_rn(y, y);
        return sq > 0.f && (1.f - sq) > 0.f ? y + y : 0.f;
    }
    const float c = (y > 0.f && (1.f - y) > 0.f) ? 1.f : 0.f;
    if (act != 2) return c;
    const float half = c * sqrtf(y);
    return half + half;
}

__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

__device__ __forceinline__ float4 scale4(float4 v, float f) { return make_float4(v.x * f, v.y * f, v.z * f, v.w * f); }

__device__ __forceinline__ void load_slots(const uint16_t* list, int nnz, int lane, uint32_t& s0, uint32_t& s1) {
    s0 = lane < nnz ? list[lane] : kNoFeature;
    s1 = lane + 32 < nnz ? list[lane + 32] : kNoFeature;
}

// ---------------------------------------------------------------- gather forward
// grid = (ceil(2n / pairs), column chunks); block = 256 threads (8 warps), a warp per pair and chunk.
// Takes index sets without block structure, and the small batches of networks that have it: staging the table's tiles
// costs the tiled kernel the whole table whatever the batch holds, here only the rows of the batch are read.
// Bound by load latency for few warps, then by the instructions around a row's loads: a warp takes up to 512 columns, and one row at a time
// leaves the registers to more warps.  Operator, 2048 positions x 1024 columns (285 MB of rows from L2, whole call, us): 128 columns a warp
// and four rows at a time 53, 256 and four 52, 256 and two 45, 256 and one 41, 512 and two 47, 512 and one 39 (rows copied ahead into a ring in
// shared memory, 512 columns: 43); 1000 x 2048 pairwise, 256 columns: four rows 69, two 44, one 50; 8192 x 128: four 34, two 31; with a factoriser
// (whole evaluation of 300 x 2048 pairwise): four rows 75, one 66.  Of few warps each needs the rows in flight: 300 x 1024 22 with four, 24 with one.
// With a factoriser the two rows of a feature are added as they arrive, so a small batch does not merge the table first.
struct GatherShape {
    int pieces, rows;  // of 128 columns that a warp takes (with the pairwise product half of them of each half), rows at a time
    int pairs;         // per CTA: one per warp while there are few, up to eight once that leaves two waves of eight CTAs per SM
    dim3 grid;
};
// Four rows at a time up to `few` warps per SM of that form.  Forward alone, us, 768 x 16 rows, four / one row at a time, half of the slots active,
// at 24, 40, 48, 56, 64, 72, 96 warps:
//   with a factoriser  x 512 columns 10 / 16, 14.2 / 16.8, 16.1 / 17.1; x 1024 16 / 24, 19.2 / 23.8, 20.4 / 24.5; x 64 7.5 / 11.8
//   without  x 512 -, 8.7 / 14.5, 12.2 / 14.5, 12.4 / 14.3, 12.5 / 14.5, 12.7 / 14.6, 15.4 / 14.8; x 1024 -, 14.2 / 21.9, 16.1 / 21.7, 17.4 / 21.8, 17.4 / 21.8,
//   17.8 / 21.5, 21.5 / 21.7; 147 rows, where the rows come sooner, x 256 54 warps 11.1 / 9.0, x 512 11.5 / 11.8, x 1024 12.4 / 13.4
// 512 columns a warp where that halves the chunks of 256: a chunk's warps take a row's latency each, however few columns they have.  Two / four pieces,
// 2048 positions, 768 rows: 320 columns 14.6 / 10.6, 448 15.6 / 11.5, 576 (three chunks or two) 17.6 / 18.2, 768 18.4 / 19.2, 896 23.2 / 20.1.
inline GatherShape gather_shape(int n, int unit, bool pairwise, bool factor, int sms) {
    const long long all = 2LL * n * ((unit + 127) / 128);
    const int few = pairwise ? factor ? 16 : 48 : factor ? 40 : unit >= 1024 ? 64 : 48;
    GatherShape g{};
    if (all < (long long)few * sms) g.pieces = pairwise ? 2 : 1, g.rows = 4;
    else if (pairwise) g.pieces = 2, g.rows = factor ? 1 : 2;
    else if (unit > 128) g.pieces = (unit + 255) / 256 == 2 * ((unit + 511) / 512) ? 4 : 2, g.rows = 1;
    else g.pieces = 1, g.rows = factor ? 1 : 2;
    const int wide = 128 * (pairwise ? g.pieces / 2 : g.pieces), chunks = (unit + wide - 1) / wide;
    const long long per = 2LL * n * chunks / (8LL * 16 * sms);
    g.pairs = 8 * (int)(per < 1 ? 1 : per < 8 ? per : 8);
    g.grid = dim3((2 * n + g.pairs - 1) / g.pairs, chunks);
    return g;
}
// C: pieces of 128 columns that a warp takes (with the pairwise product half of them of each half), U rows of them at a time.
template <bool PAIRWISE, bool FACTOR, int C, int U>
__global__ void __launch_bounds__(256) ft_forward_gather_kernel(FtArgs a, int pairs_per_block) {
    ft_step_begin(a);
    constexpr int H2 = PAIRWISE ? 2 : 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int unit = PAIRWISE ? a.H / 2 : a.H;
    const int col = blockIdx.y * (128 * C / H2) + lane * 4;
    const int pair_end = min(2 * a.n, (int)(blockIdx.x + 1) * pairs_per_block);
    auto at = [&](int c) { return 128 * (c / H2) + (c % H2 ? unit : 0); };  // piece c: of each half in turn; from this lane's column on
    bool on[C];
#pragma unroll
    for (int c = 0; c < C; c++) on[c] = col + 128 * (c / H2) < unit;
    // few warps: nothing else covers the bias's latency at the end
    constexpr bool EARLY = U == 4;
    auto bias_at = [&](int c) { return *reinterpret_cast<const float4*>(a.bias + col + at(c)); };
    float4 bias[EARLY ? C : 1];
    if (EARLY)
#pragma unroll
        for (int c = 0; c < C; c++)
            if (on[c]) bias[c] = bias_at(c);
    for (int pair = blockIdx.x * pairs_per_block + warp; pair < pair_end; pair += 8) {
        const int b = pair >> 1, p = pair & 1;
        const uint16_t* list = (p ? a.idx_nstm : a.idx_stm) + (size_t)b * a.nnz;
        uint32_t slot[2];
        load_slots(list, a.nnz, lane, slot[0], slot[1]);
        unsigned mask[2];
        mask[0] = __ballot_sync(0xffffffffu, slot[0] < (uint32_t)a.n_inputs);
        mask[1] = __ballot_sync(0xffffffffu, slot[1] < (uint32_t)a.n_inputs);
        if (a.block_rows > 0 && (mask[0] | mask[1])) {
            const uint32_t first = __shfl_sync(0xffffffffu, mask[0] ? slot[0] : slot[1], __ffs(mask[0] ? mask[0] : mask[1]) - 1);
            const uint32_t base = first / a.block_rows * a.block_rows;
            const unsigned all0 = mask[0], all1 = mask[1];
            mask[0] &= __ballot_sync(0xffffffffu, slot[0] - base < (uint32_t)a.block_rows);
            mask[1] &= __ballot_sync(0xffffffffu, slot[1] - base < (uint32_t)a.block_rows);
            if (a.status && lane == 0 && (mask[0] != all0 || mask[1] != all1)) *a.status = kStatusOutsideBlock;
        }
        const uint32_t frow[2] = {FACTOR ? slot[0] % a.factor_rows : 0u, FACTOR ? slot[1] % a.factor_rows : 0u};
        float4 sum[C];
#pragma unroll
        for (int c = 0; c < C; c++) sum[c] = make_float4(0, 0, 0, 0);
#pragma unroll
        for (int half = 0; half < 2; half++) {
            unsigned m = mask[half];
            while (m) {  // up to U rows' independent loads in flight, added in slot order
                float4 v[U][C], w[U][C];
                uint32_t f[U], ff[U];
                int cnt = 0;
#pragma unroll
                for (int k = 0; k < U; k++) {
                    const int s = m ? __ffs(m) - 1 : 0;
                    if (m) cnt++;
                    m &= m - 1;
                    f[k] = __shfl_sync(0xffffffffu, slot[half], s);
                    if (FACTOR) ff[k] = __shfl_sync(0xffffffffu, frow[half], s);
                }
#pragma unroll
                for (int k = 0; k < U; k++) {
                    const float* row = a.table + (size_t)f[k] * a.H + col;
#pragma unroll
                    for (int c = 0; c < C; c++)
                        if (k < cnt && on[c]) v[k][c] = __ldg(reinterpret_cast<const float4*>(row + at(c)));
                }
                if (FACTOR)
#pragma unroll
                    for (int k = 0; k < U; k++) {
                        const float* row = a.factor + (size_t)ff[k] * a.H + col;
#pragma unroll
                        for (int c = 0; c < C; c++)
                            if (k < cnt && on[c]) w[k][c] = __ldg(reinterpret_cast<const float4*>(row + at(c)));
                    }
#pragma unroll
                for (int k = 0; k < U; k++)
#pragma unroll
                    for (int c = 0; c < C; c++)
                        if (k < cnt && on[c]) sum[c] = add4(sum[c], FACTOR ? add4(v[k][c], w[k][c]) : v[k][c]);
            }
        }
#pragma unroll
        for (int c = 0; c < C; c += H2) {
            if (!on[c]) break;
            const float4 lo = add4(sum[c], EARLY ? bias[EARLY ? c : 0] : bias_at(c));
            if (PAIRWISE) {
                const float4 hi = add4(sum[c + H2 - 1], EARLY ? bias[EARLY ? c + H2 - 1 : 0] : bias_at(c + H2 - 1));
                const float4 ul = make_float4(crelu_f(lo.x), crelu_f(lo.y), crelu_f(lo.z), crelu_f(lo.w));
                const float4 uh = make_float4(crelu_f(hi.x), crelu_f(hi.y), crelu_f(hi.z), crelu_f(hi.w));
                float* up = a.u + (size_t)pair * a.H + col;
                *reinterpret_cast<float4*>(up + at(c)) = ul;
                *reinterpret_cast<float4*>(up + at(c + H2 - 1)) = uh;
                *reinterpret_cast<float4*>(a.x + (size_t)pair * unit + col + at(c)) = make_float4(ul.x * uh.x, ul.y * uh.y, ul.z * uh.z, ul.w * uh.w);
            } else {
                *reinterpret_cast<float4*>(a.x + (size_t)pair * a.H + col + at(c)) = make_float4(
                    ft_act_fwd(a.act, lo.x), ft_act_fwd(a.act, lo.y), ft_act_fwd(a.act, lo.z), ft_act_fwd(a.act, lo.w));
            }
        }
    }
}

typedef void (*GatherKernel)(FtArgs, int);
template <bool PAIRWISE, bool FACTOR>
GatherKernel gather_form(const GatherShape& g) {
    if (g.rows == 4) return ft_forward_gather_kernel<PAIRWISE, FACTOR, PAIRWISE ? 2 : 1, 4>;
    if (PAIRWISE) return ft_forward_gather_kernel<true, FACTOR, 2, FACTOR ? 1 : 2>;
    if (g.pieces == 4) return ft_forward_gather_kernel<false, FACTOR, 4, 1>;
    if (g.pieces == 2) return ft_forward_gather_kernel<false, FACTOR, 2, 1>;
    return ft_forward_gather_kernel<false, FACTOR, 1, FACTOR ? 1 : 2>;
}

// --------------------------------------------------------------- gather backward
// Same decomposition.  The table gradient must be zero on entry; gradients are
// added with 128-bit global reductions, the bias gradient once per lane per block.
template <bool PAIRWISE, bool ONE>
__global__ void __launch_bounds__(256) ft_backward_gather_kernel(FtArgs a, int pairs_per_block) {
    step_begin(a.stamp);
    __shared__ float4 red[2][8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int unit = PAIRWISE ? a.H / 2 : a.H;
    const int col = blockIdx.y * 128 + lane * 4;
    const bool active = col < unit;
    const int pair_end = min(2 * a.n, (int)(blockIdx.x + 1) * pairs_per_block);
    float4 bsum_lo = make_float4(0, 0, 0, 0), bsum_hi = bsum_lo;
    for (int pair = blockIdx.x * pairs_per_block + warp; pair < pair_end; pair += 8) {
        const int b = pair >> 1, p = pair & 1;
        float4 glo = make_float4(0, 0, 0, 0), ghi = glo;
        const float dout = ONE ? a.dout[b] : 0.f;
        const float* w1 = ONE ? a.w1 + (size_t)a.out_bucket[b] * 2 * unit + p * unit + col : nullptr;
        if (active) {
            if (PAIRWISE) {
                const float* up = a.u + (size_t)pair * a.H;
                const float4 ul = *reinterpret_cast<const float4*>(up + col);
                const float4 uh = *reinterpret_cast<const float4*>(up + unit + col);
                const float4 d = ONE ? scale4(__ldg(reinterpret_cast<const float4*>(w1)), dout) : *reinterpret_cast<const float4*>(a.dx + (size_t)b * a.H + (size_t)p * unit + col);
                glo = make_float4((d.x * uh.x) * ft_act_bwd(1, ul.x), (d.y * uh.y) * ft_act_bwd(1, ul.y),
                                  (d.z * uh.z) * ft_act_bwd(1, ul.z), (d.w * uh.w) * ft_act_bwd(1, ul.w));
                ghi = make_float4((d.x * ul.x) * ft_act_bwd(1, uh.x), (d.y * ul.y) * ft_act_bwd(1, uh.y),
                                  (d.z * ul.z) * ft_act_bwd(1, uh.z), (d.w * ul.w) * ft_act_bwd(1, uh.w));
            } else {
                const size_t at = (size_t)b * 2 * a.H + (size_t)p * a.H + col;
                const float4 y = *reinterpret_cast<const float4*>(a.x + at);
                const float4 d = ONE ? scale4(__ldg(reinterpret_cast<const float4*>(w1)), dout) : *reinterpret_cast<const float4*>(a.dx + at);
                glo = make_float4(d.x * ft_act_bwd(a.act, y.x), d.y * ft_act_bwd(a.act, y.y),
                                  d.z * ft_act_bwd(a.act, y.z), d.w * ft_act_bwd(a.act, y.w));
            }
        }
        const bool lo_nz = glo.x != 0.f || glo.y != 0.f || glo.z != 0.f || glo.w != 0.f;
        const bool hi_nz = PAIRWISE && (ghi.x != 0.f || ghi.y != 0.f || ghi.z != 0.f || ghi.w != 0.f);
        if (!__any_sync(0xffffffffu, lo_nz || hi_nz)) continue;  // the reference skips zero gradients too
        bsum_lo = add4(bsum_lo, glo);
        bsum_hi = add4(bsum_hi, ghi);
        const uint16_t* list = (p ? a.idx_nstm : a.idx_stm) + (size_t)b * a.nnz;
        uint32_t slot[2];
        load_slots(list, a.nnz, lane, slot[0], slot[1]);
#pragma unroll
        for (int half = 0; half < 2; half++) {
            unsigned m = __ballot_sync(0xffffffffu, slot[half] < (uint32_t)a.n_inputs);
            while (m) {
                const int s = __ffs(m) - 1;
                m &= m - 1;
                const uint32_t f = __shfl_sync(0xffffffffu, slot[half], s);
                float* row = a.g_table + (size_t)f * a.H;
                if (lo_nz) atomicAdd(reinterpret_cast<float4*>(row + col), glo);
                if (hi_nz) atomicAdd(reinterpret_cast<float4*>(row + unit + col), ghi);
            }
        }
    }
    red[0][warp][lane] = bsum_lo;
    red[1][warp][lane] = bsum_hi;
    __syncthreads();
    if (warp == 0 && active) {
        float4 s_lo = red[0][0][lane], s_hi = red[1][0][lane];
        for (int w = 1; w < 8; w++) {
            s_lo = add4(s_lo, red[0][w][lane]);
            s_hi = add4(s_hi, red[1][w][lane]);
        }
        atomicAdd(reinterpret_cast<float4*>(a.g_bias + col), s_lo);
        if (PAIRWISE) atomicAdd(reinterpret_cast<float4*>(a.g_bias + unit + col), s_hi);
    }
}

// ------------------------------------------------------------------ tiled kernels
// A tile row holds 64 floats of one table row; lane l of a half warp owns floats 4l to 4l + 3 and
// moves them with one 16-byte shared-memory access and two packed f32x2 adds.  Without pairwise
// they are neighbouring columns, 64s + 4l on; with pairwise the low-half columns 32s + 2l and 32s + 2l + 1,
// each before its partner H/2 further on, i.e. both factors of two products.
constexpr int kTileCols = 64;
constexpr int kTileRowBytes = kTileCols * 4;

typedef unsigned long long f32x2;  // two packed floats: low word = A, high word = B

__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {  // two IEEE fp32 adds in one instruction
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    return (f32x2)__float_as_uint(a) | ((f32x2)__float_as_uint(b) << 32);
}
__device__ __forceinline__ float lo2(f32x2 v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float hi2(f32x2 v) { return __uint_as_float((unsigned)(v >> 32)); }

// Loads of data that is read once per kernel and must not claim L1 lines: with 196-228 KB of the SM's 256 KB
// configured as shared memory only 28-60 KB of L1 are left, less than these kernels keep in flight.
// ld_fresh4: what the kernel before wrote, which may still be writing when this one begins (launch.cuh).
__device__ __forceinline__ float4 ld_once4(const float4* p) {
    float4 v;
    asm("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 ld_fresh4(const float4* p) {
    float4 v;
    asm volatile("ld.global.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// The row walks take a line with 16 lanes and 16 bytes each, so that a warp serves two lists at a time: lane l owns floats
// 4 (l mod 16) .. + 3 of the line.  A list entry is a 16-bit line index; one byte permutation turns it into the byte offset
// of this lane's piece, because a line is 256 bytes and `lane16` = 16 (l mod 16) fills exactly the lowest byte.
__device__ __forceinline__ uint32_t entry_lo(uint32_t word, uint32_t lane16) { return __byte_perm(word, lane16, 0x5104); }
__device__ __forceinline__ uint32_t entry_hi(uint32_t word, uint32_t lane16) { return __byte_perm(word, lane16, 0x5324); }
struct f32x4 {  // four floats as two packed pairs
    f32x2 a, b;
};
__device__ __forceinline__ f32x4 quad_at(const unsigned char* lines, uint32_t offset) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(lines + offset);
    return {v.x, v.y};
}
__device__ __forceinline__ f32x4 add2(f32x4 x, f32x4 y) { return {add2(x.a, y.a), add2(x.b, y.b)}; }
// Sum of the lines that `len` entries at `list` (shared memory, 8-byte aligned) name, added in list order from +0.  Four
// entries per 8-byte load, fetched one group ahead (up to 16 bytes past the list's last group are read and not used);
// the lanes of a half warp agree on list and length, the two halves need not.  (Not unrolled: the compiler's own choice cost the forward 1549 against
// 1505 us at 131072 positions x 2048 columns, 232 against 228 at 16384, 118 against 114 at 1024 columns; by two 1522, 229, 114.5; by four 1530, 229, 115.)
__device__ __forceinline__ f32x4 sum_lines(const unsigned char* lines, const uint2* list, int len, uint32_t lane16) {
    f32x4 acc = {0, 0};
    uint2 g = *list;
#pragma unroll 1
    for (len -= 4; len >= 0; len -= 4) {
        const uint2 ahead = *++list;
        const f32x4 v0 = quad_at(lines, entry_lo(g.x, lane16)), v1 = quad_at(lines, entry_hi(g.x, lane16));
        const f32x4 v2 = quad_at(lines, entry_lo(g.y, lane16)), v3 = quad_at(lines, entry_hi(g.y, lane16));
        acc = add2(add2(add2(add2(acc, v0), v1), v2), v3);
        g = ahead;
    }
    const int rest = len + 4;  // none to three more
    if (rest > 0) {
        acc = add2(acc, quad_at(lines, entry_lo(g.x, lane16)));
        if (rest > 1) acc = add2(acc, quad_at(lines, entry_hi(g.x, lane16)));
        if (rest > 2) acc = add2(acc, quad_at(lines, entry_lo(g.y, lane16)));
    }
    return acc;
}

// The same for lists of an even length, whose last entry may be a line of zeros: the backward's pieces are short (11 entries at 512 pairs
// of a 768-row block), and up to three single lines at their ends cost more instructions than the added half line costs passes through
// the pipe (2048 columns pairwise, 16384 positions 282 -> 270 us, 131072 1974 -> 1900).  The forward's longer lists lose by it (231 -> 240 at 16384,
// 147 rows 70.6 -> 73.3).
// TWO: the loop unrolled by two groups of four, which helps the backward without the pairwise product (1024 columns 142 -> 137 us), whose
// warps have the registers, and hurts it with the product (the same sizes 267 -> 270, 1847 -> 1871; not unrolled at all 274, 1905).
template <bool TWO>
__device__ __forceinline__ f32x4 sum_lines_even(const unsigned char* lines, const uint2* list, int len, uint32_t lane16) {
    f32x4 acc = {0, 0};
    uint2 g = *list;
    auto four = [&]() {
        const uint2 ahead = *++list;
        const f32x4 v0 = quad_at(lines, entry_lo(g.x, lane16)), v1 = quad_at(lines, entry_hi(g.x, lane16));
        const f32x4 v2 = quad_at(lines, entry_lo(g.y, lane16)), v3 = quad_at(lines, entry_hi(g.y, lane16));
        acc = add2(add2(add2(add2(acc, v0), v1), v2), v3);
        g = ahead;
    };
    len -= 4;
    if (TWO) {
#pragma unroll 2
        for (; len >= 0; len -= 4) four();
    } else {
        for (; len >= 0; len -= 4) four();
    }
    if (len == -2) {
        const f32x4 v0 = quad_at(lines, entry_lo(g.x, lane16)), v1 = quad_at(lines, entry_hi(g.x, lane16));
        acc = add2(add2(acc, v0), v1);
    }
    return acc;
}

template <bool ANY>
__device__ __forceinline__ void store_piece(float* p, float2 v) {
    if (ANY) p[0] = v.x, p[1] = v.y;
    else *reinterpret_cast<float2*>(p) = v;
}
template <bool ANY>
__device__ __forceinline__ void store_piece(float* p, float4 v) {
    if (ANY) p[0] = v.x, p[1] = v.y, p[2] = v.z, p[3] = v.w;
    else *reinterpret_cast<float4*>(p) = v;
}

// Forward.  One CTA of 1024 threads per SM; dynamic shared memory = R tile rows, then per warp two prepared lists (and 16
// bytes that a read-ahead may touch).  A CTA walks its piece of the work line segment by segment; a segment is a run of
// pairs of one (block, slab), whose tile the CTA loads first.  Each warp serves two neighbouring pairs at a time, one per
// half warp; the grouping has put lists of nearly the same length side by side.  The lists reach the warp one round ahead:
// the lanes load them as 32-bit words into registers while the pairs before are still being walked, and store them into the
// warp's buffer afterwards, so the walk itself reads no global memory.  Every lane adds its four columns with one 16-byte
// shared-memory load and two packed adds per row, in slot order — the same order and arithmetic as the interpreter.
// AHEAD: while a tile is walked the next one is fetched into tensor memory (64 columns of 32 lanes for each warp, which no other
// warp touches), and copied from there when all warps have left the tile.  Fetched only then it kept the pipe idle for 26 k of 105 k clocks
// per tile at 16384 positions (2048 columns pairwise: 262 against 231 us).  Each warp fetches its share in one go, with the registers of the walk free, the warps
// one after the other; a piece of it in every round instead, held in registers through the walk, cost the walk more than it saved at 131072.
// Bound by the shared-memory pipe: 256 bytes per (row, pair, slab) at 128 bytes a clock.  (One pair per warp, 8 bytes per
// lane, spent twice the instructions per row and was bound by their issue: 1.69 against 1.55 ms at 131072 positions and
// width 2048, 0.273 against 0.260 ms at 16384.)
constexpr int kFwdThreads = 1024;
// Tables of up to about 900 rows: the tile and two lists for each of 16 warps at least must fit.
__host__ __device__ inline bool ft_fwd_fits(int R, int list_len) {
    return (size_t)(R + 1) * kTileRowBytes + (size_t)(kFwdThreads / 32) * list_len * 2 + 16 <= 227 * 1024;
}
// Warps that walk lists: all of them, or (the last few rows of that range) as many as have room for two lists beside the tile.
__host__ __device__ inline int ft_fwd_warps(int R, int list_len) {
    const int room = (227 * 1024 - 16 - R * kTileRowBytes) / (list_len * 4);
    return room < kFwdThreads / 32 ? room : kFwdThreads / 32;
}
__host__ __device__ inline size_t ft_fwd_smem(int R, int list_len) {
    return (size_t)R * kTileRowBytes + (size_t)ft_fwd_warps(R, list_len) * list_len * 4 + 16;
}

// Whether the CTAs of a launch fetch a next tile while they walk (AHEAD): where many of them have one, and rounds enough to fetch it in.
// Forward on a B200, without / with, us: 768 x 16 rows, 16384 positions, 2048 columns pairwise 252 / 231, 131072 positions 1547 / 1549,
// 1024 columns 136 / 132, 256 columns 39 / 39; 625 pairs a tile (5003 x 512) 40.3 / 39.2, but no gain in the whole pass; 375 (3000 x 64)
// 16.5 / 18.5, 188 (1500 x 2048) 46 / 48; two tiles in all (768 rows x 128 columns) 20.8 / 21.2.
inline bool ft_fwd_ahead(const FtArgs& a, const TileArgs& t, int grid) {
    const long long pairs_per_tile = 2LL * a.n / (a.n_inputs / t.block_rows);
    return 2LL * t.nslabs * (t.last_block - t.first_block) > grid && pairs_per_tile >= 1024;
}

// ANY: bias, x and u start on any float (the operator's caller owns them); else on 8 bytes with the pairwise product, on 16
// without, and move in pieces of that size.
template <bool PAIRWISE, bool AHEAD, bool ANY = false>
__global__ void __launch_bounds__(kFwdThreads, 1) ft_forward_tiled_kernel(FtArgs a, TileArgs t) {
    ft_step_begin(a);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int NW = t.walk_warps;
    const int R = t.block_rows, half = lane >> 4, l16 = lane & 15;
    const uint32_t lane16 = 16 * l16;
    float* tile = reinterpret_cast<float*>(smem_raw);
    // outputs of pair p start at p * (row length): x is [n][2 persp][H or H/2], u is [n][2][H]
    const int x_row = PAIRWISE ? a.H / 2 : a.H;
    const int words = t.list_len;  // 32-bit words of two lists
    uint32_t* ring = reinterpret_cast<uint32_t*>(smem_raw + (size_t)R * kTileRowBytes) + warp * words;
    const uint2* list = reinterpret_cast<const uint2*>(ring + half * (words / 2));
    const uint32_t* lists_w = reinterpret_cast<const uint32_t*>(t.lists);
    // This CTA's piece of the line of nslabs x (pairs of the launch's blocks) positions is walked in segments, runs of pairs of
    // one tile.  `rest`: pairs from the segment's first one on; the segments after the first start at their tile's first pair.
    int block = t.first_block, slab = 0, first, rest;
    {
        const int pair0 = t.block_begin[block];
        const long long line = (long long)t.nslabs * (t.block_begin[t.last_block] - pair0), v = line * blockIdx.x / gridDim.x;
        rest = (int)(line * (blockIdx.x + 1) / gridDim.x - v);
        if (rest <= 0) return;
        long long at = v;
        int in_block = t.block_begin[block + 1] - pair0;
        while (at >= (long long)t.nslabs * in_block) {
            at -= (long long)t.nslabs * in_block;
            block++;
            in_block = t.block_begin[block + 1] - t.block_begin[block];
        }
        slab = (int)(at / in_block);
        first = t.block_begin[block] + (int)(at - (long long)slab * in_block);
    }
    auto next_tile = [&](int& block, int& slab) {
        if (++slab < t.nslabs) return;
        slab = 0;
        do block++;
        while (t.block_begin[block + 1] == t.block_begin[block]);
    };
    // A tile's rows are filled in by eight threads each, two 16-byte pieces of a thread that its neighbours continue.
    // With a factoriser the table row is l0w[row] + l0f[row mod factor_rows], one fp32 add per element exactly as the
    // reference forms `l0w + l0f.repeat(n)` (model/builder.rs:421-424).
    const int q = threadIdx.x & 7, row0 = threadIdx.x >> 3;
    constexpr int kFillRows = kFwdThreads / 8;
    auto fill = [&](int block, int slab, auto put) {
        const float* src = a.table + (size_t)block * R * a.H;
        const int c0 = PAIRWISE ? slab * 32 + q * 4 : slab * 64 + q * 4, c1 = PAIRWISE ? a.H / 2 + c0 : c0 + 32;
        const bool in0 = c0 < x_row, in1 = PAIRWISE ? in0 : c1 < x_row;  // the last slab of a width that 64 does not divide
#pragma unroll 3
        for (int step = 0; step < t.fill_steps; step++) {
            const int row = row0 + step * kFillRows;
            float4 v0 = make_float4(0, 0, 0, 0), v1 = v0;
            if (row < R) {
                if (in0) v0 = ld_once4(reinterpret_cast<const float4*>(src + (size_t)row * a.H + c0));
                if (in1) v1 = ld_once4(reinterpret_cast<const float4*>(src + (size_t)row * a.H + c1));
                if (a.factor) {
                    const float* frow = a.factor + (size_t)((block * R + row) % a.factor_rows) * a.H;
                    if (in0) v0 = add4(v0, __ldg(reinterpret_cast<const float4*>(frow + c0)));
                    if (in1) v1 = add4(v1, __ldg(reinterpret_cast<const float4*>(frow + c1)));
                }
            }
            put(step, row, v0, v1);
        }
    };
    auto put_row = [&](int row, const float4& v0, const float4& v1) {
        float4* dst = reinterpret_cast<float4*>(tile + row * kTileCols);
        if (PAIRWISE) {
            // the tile row holds (low-half column, its high-half partner) side by side, both factors of one product.
            // (A thread's pieces lie next to each other, 32 bytes from its neighbour's: the upper four threads of a
            // row store their second piece first, so that the eight stores of a quarter warp fall into eight
            // different bank groups)
            const int h = q >> 2;
            const float4 first4 = make_float4(v0.x, v1.x, v0.y, v1.y), second4 = make_float4(v0.z, v1.z, v0.w, v1.w);
            dst[2 * q + h] = h ? second4 : first4;
            dst[2 * q + (h ^ 1)] = h ? first4 : second4;
        } else {
            dst[q] = v0;
            dst[q + 8] = v1;
        }
    };
    const uint32_t spare = tmem_own(warp, 64);
    bool filled = false;
    for (;;) {
        const int seg_end = min(t.block_begin[block + 1], first + rest);
        rest -= seg_end - first;
        int i = warp < NW ? first + 2 * warp : seg_end;
        int2 next = make_int2(0, 0);  // this half's next pair and its length
        uint32_t w0 = 0, w1 = 0;      // this lane's words of the next two lists
        auto fetch = [&](int at) {
            if (at + half < seg_end) next = t.pairs[at + half];
            // (a single last pair: the second list of the two may lie past the end of the lists)
            const int have = at + 1 < seg_end ? words : words / 2;
            const uint32_t* src = lists_w + (size_t)at * (words / 2);
            if (at < seg_end && lane < have) w0 = src[lane];
            if (at < seg_end && lane + 32 < have) w1 = src[lane + 32];
        };
        fetch(i);
        if (AHEAD && !filled && rest > 0 && warp == 0) tmem_alloc_all(ring);  // (the word is not needed, the lists come later)
        __syncthreads();  // every warp has left the previous tile
        if (AHEAD && filled) {
            tmem_stored();
            for (int row = row0, at = 0; at < t.fill_steps; row += kFillRows, at++) {
                float4 v0, v1;
                tmem_get8(spare + 8 * at, v0, v1);
                if (row < R) put_row(row, v0, v1);
            }
        } else {
            fill(block, slab, [&](int step, int row, const float4& v0, const float4& v1) {
                if (row < R) put_row(row, v0, v1);
            });
        }
        // this lane's columns: two products, or four neighbours
        const int col = PAIRWISE ? slab * 32 + 2 * l16 : slab * 64 + 4 * l16;
        f32x4 bias = {0, 0};
        const bool col_on = col < x_row;
        if (!col_on) {
        } else if (ANY) {
            const float* b = a.bias + col;
            bias = PAIRWISE ? f32x4{pack2(b[0], b[a.H / 2]), pack2(b[1], b[a.H / 2 + 1])} : f32x4{pack2(b[0], b[1]), pack2(b[2], b[3])};
        } else if (PAIRWISE) {
            const float2 lo = *reinterpret_cast<const float2*>(a.bias + col), hi = *reinterpret_cast<const float2*>(a.bias + a.H / 2 + col);
            bias = {pack2(lo.x, hi.x), pack2(lo.y, hi.y)};
        } else {
            const float4 b = *reinterpret_cast<const float4*>(a.bias + col);
            bias = {pack2(b.x, b.y), pack2(b.z, b.w)};
        }
        float* x_out = a.x + col;
        __syncthreads();
        auto round = [&]() {
            const int pair = next.x, cnt = i + half < seg_end ? next.y : 0;
            __syncwarp();  // every lane has finished with the lists of the pairs before
            if (lane < words) ring[lane] = w0;
            if (lane + 32 < words) ring[lane + 32] = w1;
            fetch(i + 2 * NW);
            __syncwarp();
            const f32x4 acc = add2(sum_lines(smem_raw, list, cnt, lane16), bias);
            if (i + half < seg_end && col_on) {
                if (PAIRWISE) {
                    const float2 ulo = make_float2(crelu_f(lo2(acc.a)), crelu_f(lo2(acc.b))), uhi = make_float2(crelu_f(hi2(acc.a)), crelu_f(hi2(acc.b)));
                    float* up = a.u + (size_t)pair * a.H + col;
                    store_piece<ANY>(up, ulo);
                    store_piece<ANY>(up + a.H / 2, uhi);
                    store_piece<ANY>(x_out + (size_t)pair * x_row, make_float2(ulo.x * uhi.x, ulo.y * uhi.y));
                } else {
                    store_piece<ANY>(
                        x_out + (size_t)pair * x_row,
                        make_float4(ft_act_fwd(a.act, lo2(acc.a)), ft_act_fwd(a.act, hi2(acc.a)), ft_act_fwd(a.act, lo2(acc.b)), ft_act_fwd(a.act, hi2(acc.b))));
                }
            }
            i += 2 * NW;
        };
        if (AHEAD && rest > 0) {
            const int turn = i + (seg_end - first) / (2 * NW) * warp / 32 * 2 * NW;
            while (i < min(turn, seg_end)) round();
            __syncwarp();
            int next_block = block, next_slab = slab;
            next_tile(next_block, next_slab);
            fill(next_block, next_slab, [&](int step, int row, const float4& v0, const float4& v1) { tmem_put8(spare + 8 * step, v0, v1); });
            filled = true;
        }
        while (i < seg_end) round();
        if (rest == 0) break;
        next_tile(block, slab);
        first = t.block_begin[block];
    }
    if (AHEAD && filled && warp == 0) tmem_free_all();  // (every access lies before the last tile's barrier)
}

// Backward.  Positions are visited in chunks of at most CP pairs of one row block.
//   ft_csr_kernel (one CTA per chunk, once per batch) turns the chunk's prepared lists around:
//     for every table row of the block, the list of the chunk's pairs that hold it (a count,
//     a scan and a fill in shared memory), every list starting on an 8-byte
//     boundary.  Lists are cut into pieces of at most kPiece entries and the pieces put in
//     order of their lengths, longest first.  All column slabs share the result.
//   ft_backward_tiled_kernel (same grid as the forward) then, per chunk, copies that list
//     structure into shared memory, stages the chunk's pre-activation gradients (from dx and
//     the kept activations) as one 64-float line per pair, and every half warp walks pieces,
//     sums the staged lines in registers and adds the total to the row of the table gradient
//     with one 16-byte global reduction per lane.
// Accumulation needs no atomics, and the table gradient sees one reduction per (row piece, chunk)
// instead of one per (row, position).  The table gradient must be zero on entry.
constexpr int kCsrThreads = 1024;

// Two shapes of the backward: "wide" = one CTA of 1024 threads per SM, otherwise two CTAs of 512 threads on chunks of 256
// pairs (half of it when nnz > 32), so that one CTA's global loads overlap the other's shared-memory work.
constexpr int kChunkLeast = 128, kChunkMost = 640;  // pairs per chunk of the wide shape
__host__ __device__ inline int ft_bwd_chunk_narrow(int nnz) { return nnz <= 32 ? 256 : 128; }
// Most entries of a piece: the pieces of a chunk differ in length by little from one warp's next to another's, and a king's
// row, which half the pairs of a chunk may hold, is shared out.
constexpr int kPiece = 64;
// entries per chunk: every slot of every pair plus up to three unused ones per row (lists start on 8 bytes), and 16 bytes
// that a read-ahead may touch
__host__ __device__ inline int ft_bwd_ent_cap(int R, int nnz, int cp) { return (cp * nnz + 4 * R + 8 + 7) & ~7; }
// per chunk: entries, pieces, two unused words, then the pieces: first entry / 4 << 17 | length, rounded up to even << 10 | row
__host__ __device__ inline int ft_bwd_start_cap(int R, int nnz, int cp) { return (4 + R + cp * nnz / kPiece + 3) & ~3; }
__host__ __device__ inline size_t ft_bwd_smem(int R, int nnz, int cp) {
    return (size_t)(cp + 1) * kTileRowBytes + (size_t)ft_bwd_ent_cap(R, nnz, cp) * 2 + (size_t)ft_bwd_start_cap(R, nnz, cp) * 4 + (size_t)cp * 12 +
           32 * kTileRowBytes;  // staged lines, row lists, their pieces, what a pair needs, bias-gradient sums per warp
}
__host__ __device__ inline size_t ft_csr_smem(int R, int nnz, int cp) {
    return (size_t)ft_bwd_ent_cap(R, nnz, cp) * 2 + (size_t)(2 * (R + 2)) * 4;
}

// grid = most chunks there can be, block = kCsrThreads.  Bound by latency: one load of the lists, whose entries and ranks stay
// in registers from the count to the fill (a second pass over them, with a second atomic each, made it 15 us instead of
// 8.7 for chunks of 443 pairs; while a step runs, a CTA of this kernel holds up whatever kernel of the step wants its SM).
static __global__ void __launch_bounds__(kCsrThreads) ft_csr_kernel(FtArgs a, TileArgs t) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int warp_tot[32], bin[kPiece + 1];  // bin: pieces by length, then their first places
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int4 chunk = t.chunks[blockIdx.x];
    if (chunk.z == 0) return;  // (the launch is sized from the batch size alone)
    const int R = t.block_rows, c0 = chunk.y, cn = chunk.z, Q = t.list_len / 8;  // 16-byte pieces per list
    uint16_t* ent = reinterpret_cast<uint16_t*>(smem_raw);
    int* start = reinterpret_cast<int*>(ent + t.ent_cap);  // [R + 1]
    int* count = start + R + 2;                             // [R]
    constexpr int V = (kChunkMost * 8 + kCsrThreads - 1) / kCsrThreads;
    uint4 list[V];
    int pair[V], len[V];  // of each piece: its pair and how many of its eight entries count
#pragma unroll
    for (int v = 0; v < V; v++) {
        const int e = threadIdx.x + v * kCsrThreads;
        len[v] = 0;
        if (e < cn * Q) {
            pair[v] = e / Q;
            const int q = e - pair[v] * Q;
            list[v] = __ldg(reinterpret_cast<const uint4*>(t.lists + (size_t)(c0 + pair[v]) * t.list_len) + q);
            len[v] = __ldg(&t.pairs[c0 + pair[v]].y) - 8 * q;
        }
    }
    for (int r = threadIdx.x; r < R; r += kCsrThreads) count[r] = 0;
    if (threadIdx.x <= kPiece) bin[threadIdx.x] = 0;
    __syncthreads();
    // count how often each row occurs in the chunk; an entry's rank among its row's is what the counter held
    uint32_t rank[V][4];
#pragma unroll
    for (int v = 0; v < V; v++) {
        const uint32_t w[4] = {list[v].x, list[v].y, list[v].z, list[v].w};
#pragma unroll
        for (int h = 0; h < 4; h++) {
            rank[v][h] = 0;
            if (2 * h < len[v]) rank[v][h] = (uint32_t)atomicAdd(&count[w[h] & 0xffffu], 1);
            if (2 * h + 1 < len[v]) rank[v][h] |= (uint32_t)atomicAdd(&count[w[h] >> 16], 1) << 16;
        }
    }
    __syncthreads();
    // exclusive scan of the row counts, each rounded up to a multiple of four entries (8 bytes); R is less than the threads
    static_assert(kCsrThreads >= 1023, "a thread per row");
    const int r = threadIdx.x, mine = r < R ? count[r] : 0, room = (mine + 3) & ~3;
    int incl = room;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int n = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += n;
    }
    if (lane == 31) warp_tot[warp] = incl;
    if (mine >= kPiece) atomicAdd(&bin[kPiece], mine / kPiece);
    if (mine % kPiece) atomicAdd(&bin[mine % kPiece], 1);
    __syncthreads();
    const int before = __reduce_add_sync(0xffffffffu, lane < warp ? warp_tot[lane] : 0), total = __reduce_add_sync(0xffffffffu, warp_tot[lane]);
    const int first = before + incl - room;
    if (r < R) start[r] = first;
    if (mine & 1) ent[first + mine] = (uint16_t)t.chunk_len;  // (there is room: lists are walked in pairs, the line past the chunk's is zero)
    if (warp == 0) {  // places of the pieces, longest first
        int run = 0;
        for (int base = kPiece; base > 0; base -= 32) {
            const int own = bin[base - lane];
            int sum = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int n = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += n;
            }
            bin[base - lane] = run + sum - own;
            run += __shfl_sync(0xffffffffu, sum, 31);
        }
        if (lane == 0) bin[0] = run;  // (no piece is empty: the place of length 0 holds their number)
    }
    __syncthreads();
    // fill: entry = index of the pair within the chunk, grouped by row; and the list pieces
#pragma unroll
    for (int v = 0; v < V; v++) {
        const uint32_t w[4] = {list[v].x, list[v].y, list[v].z, list[v].w};
#pragma unroll
        for (int h = 0; h < 4; h++) {
            if (2 * h < len[v]) ent[start[w[h] & 0xffffu] + (rank[v][h] & 0xffffu)] = (uint16_t)pair[v];
            if (2 * h + 1 < len[v]) ent[start[w[h] >> 16] + (rank[v][h] >> 16)] = (uint16_t)pair[v];
        }
    }
    int* out = t.csr_start + (size_t)blockIdx.x * t.start_cap;
    if (threadIdx.x == 0) *reinterpret_cast<int4*>(out) = make_int4(total, bin[0], 0, 0);
    for (int k = 0; k < mine; k += kPiece) {
        const int n = min(kPiece, mine - k);
        out[4 + atomicAdd(&bin[n], 1)] = ((first + k) >> 2) << 17 | ((n + 1) & ~1) << 10 | r;
    }
    __syncthreads();
    uint4* ent_out = reinterpret_cast<uint4*>(t.csr_ent + (size_t)blockIdx.x * t.ent_cap);
    for (int i = threadIdx.x; i < (total + 7) / 8; i += kCsrThreads) ent_out[i] = reinterpret_cast<const uint4*>(ent)[i];
}

// The backward's work line: block b contributes, per column slab, its pairs plus a fixed amount per chunk
// (the one reduction per row costs about as much as this many pairs).  A unit is one (chunk, slab);
// units are numbered chunk by chunk, and slab by slab INSIDE a chunk: a CTA that takes
// consecutive units keeps the chunk's row lists (which do not depend on the slab) in shared memory for all
// slabs, and reads neighbouring 128- or 256-byte pieces of the same activation rows from one unit to the next.
constexpr int kChunkFixed = 96;
// The units [x, y) of CTA `k` of `parts`, counted from the launch's first chunk: those between the k-th and the (k+1)-th of
// `parts` equal cuts of the line.  A whole warp, a lane per block, so that the blocks' tables cost one load latency.
__device__ __forceinline__ int2 ft_bwd_units(const TileArgs& t, int k, int parts, int lane) {
    long long line = 0;
    for (int b0 = t.first_block; b0 < t.last_block; b0 += 32) {
        const int b = b0 + lane;
        int w = 0;
        if (b < t.last_block) w = t.block_begin[b + 1] - t.block_begin[b] + kChunkFixed * (t.chunk_begin[b + 1] - t.chunk_begin[b]);
        line += __reduce_add_sync(0xffffffffu, w);
    }
    line *= t.nslabs;
    // (rounded up: units that divide evenly over the CTAs must not fall just short of their cut)
    const long long cut[2] = {(line * k + parts - 1) / parts, (line * (k + 1) + parts - 1) / parts};
    int unit[2] = {-1, -1};
    long long base = 0;
    int units = 0;
    for (int b0 = t.first_block; b0 < t.last_block; b0 += 32) {
        const int b = b0 + lane;
        int nch = 0, w = 0;
        if (b < t.last_block) {
            nch = t.chunk_begin[b + 1] - t.chunk_begin[b];
            w = t.block_begin[b + 1] - t.block_begin[b] + kChunkFixed * nch;
        }
        int w_incl = w, c_incl = nch;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int wu = __shfl_up_sync(0xffffffffu, w_incl, o), cu = __shfl_up_sync(0xffffffffu, c_incl, o);
            if (lane >= o) w_incl += wu, c_incl += cu;
        }
        const long long first = base + (long long)t.nslabs * (w_incl - w);
        for (int e = 0; e < 2; e++) {
            const bool here = nch > 0 && cut[e] >= first && cut[e] < first + (long long)t.nslabs * w;
            int at = 0;
            if (here) {  // a block's chunks are of equal size, so its units weigh the same
                const long long j = (cut[e] - first) * nch / w;
                at = units + t.nslabs * (c_incl - nch) + (int)(j < (long long)t.nslabs * nch - 1 ? j : (long long)t.nslabs * nch - 1);
            }
            const unsigned m = __ballot_sync(0xffffffffu, here);
            if (m) unit[e] = __shfl_sync(0xffffffffu, at, __ffs(m) - 1);
        }
        base += (long long)t.nslabs * __shfl_sync(0xffffffffu, w_incl, 31);
        units += t.nslabs * __shfl_sync(0xffffffffu, c_incl, 31);
    }
    return make_int2(unit[0] < 0 ? units : unit[0], unit[1] < 0 ? units : unit[1]);
}

// grid = one CTA of 1024 threads per SM (or two of 512); CTA k takes the units between the k-th and
// the (k+1)-th of gridDim.x equal cuts of the work line.  With SIGNAL (data-parallel runs whose exchange
// takes finished row blocks while this kernel is still running) the blocks must finish one after the
// other, not all at the end: CTA k then takes the units k, k + gridDim.x, ... of the block-ordered
// numbering, so that all CTAs move through the blocks together, and announces a block it has left after
// the staging phase of its next unit, when that block's reductions have had time to land (the fence
// that must precede the announcement then finds little to wait for).
//
// Staging: a pair's line takes 8 lanes (pairwise: 32 columns of each half of the accumulator) or 16 lanes, 16 bytes per
// load, the operands of the next pairs but one under way while a pair's are used (two pairs' operands a lane: more of them make the
// compiler spill).  Walk: a half warp per list piece (see sum_lines_even).  Bound by the instructions around the rows and the latency of
// shared memory in the walk (256 bytes per (row, pair, slab); the pipe is busy 70 to 75 % of it) and by load latency in the staging.  (One row per warp with 8 bytes per lane, rows in table order: 2.29 against 1.97 ms at 131072
// positions and width 2048, 0.332 against 0.281 ms at 16384.)
template <bool PAIRWISE, int THREADS, bool SIGNAL, bool ONE>
__global__ void __launch_bounds__(THREADS, 2048 / (2 * THREADS)) ft_backward_tiled_kernel(FtArgs a, TileArgs t) {
    step_begin(a.stamp);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int kBwdThreads = THREADS;
    constexpr int NW = kBwdThreads / 32;
    const int R = t.block_rows, CP = t.chunk_len;
    float* g_s = reinterpret_cast<float*>(smem_raw);                                       // [CP][64] staged lines
    uint16_t* ent = reinterpret_cast<uint16_t*>(smem_raw + (size_t)(CP + 1) * kTileRowBytes);    // lists of the chunk
    int* start = reinterpret_cast<int*>(ent + t.ent_cap);                                  // entries, pieces, -, -, then the pieces
    int* pairs_s = start + t.start_cap;                                                    // [CP] pair ids of the chunk
    float* bias_s = reinterpret_cast<float*>(pairs_s + CP);                                // [warps][64] bias-gradient sums of a unit
    int2* one_s = reinterpret_cast<int2*>(bias_s + NW * kTileCols);                        // ONE: [CP] (loss gradient, first weight) of the pair
    if (threadIdx.x < kTileCols) g_s[CP * kTileCols + threadIdx.x] = 0.f;
    const int first_chunk = t.chunk_begin[t.first_block];
    const int2 mine = SIGNAL ? make_int2(blockIdx.x, t.nslabs * (t.chunk_begin[t.last_block] - first_chunk)) : ft_bwd_units(t, blockIdx.x, gridDim.x, lane);

    // lanes of a warp per staged pair, and the four floats of the line that a lane holds: with pairwise the line is the 32
    // low-half columns, then the 32 high-half ones, so that a lane of the walk owns four neighbouring columns of the table
    constexpr int kLanes = PAIRWISE ? 8 : 16, kPairsPerWarp = 32 / kLanes;
    const int q = lane % kLanes, sub = lane / kLanes;
    const int l16 = lane & 15, half = lane >> 4;
    const uint32_t lane16 = 16 * l16;

    // Bias gradient: a warp leaves the sums of the pairs it staged in its line of bias_s; during the walk two warps add the
    // lines up, a thread per column, and reduce the result to global memory.  (Shared-memory float atomics in their place
    // took an eighth of all passes through the shared-memory pipe.)
    // staging: this lane's operands of U pairs on their way
    constexpr int U = 2, kStep = NW * kPairsPerWarp;
    float4 y0[U], y1[U], d[U];
    const int x_row = PAIRWISE ? a.H / 2 : a.H;  // columns of x per perspective
    auto fetch_one = [&](int k, int pl, int sl) {
        const int col = PAIRWISE ? sl * 32 + 4 * q : sl * 64 + 4 * q;
        if (col >= x_row) {  // the last slab of a width that 64 does not divide
            y0[k] = y1[k] = d[k] = make_float4(0, 0, 0, 0);
            return;
        }
        const int pair = pairs_s[pl];
        const float* y = (PAIRWISE ? a.u : a.x) + (size_t)pair * a.H + col;
        y0[k] = ld_once4(reinterpret_cast<const float4*>(y));
        if (PAIRWISE) y1[k] = ld_once4(reinterpret_cast<const float4*>(y + a.H / 2));
        d[k] = ONE ? __ldg(reinterpret_cast<const float4*>(a.w1 + one_s[pl].y + col))
                   : ld_fresh4(reinterpret_cast<const float4*>(a.dx + (size_t)pair * x_row + col));
    };
    auto fetch = [&](int pl0, int cn, int sl) {
#pragma unroll
        for (int k = 0; k < U; k++)
            if (pl0 + k * kStep < cn) fetch_one(k, pl0 + k * kStep, sl);
    };
    bool fetched = false;  // the unit before has fetched this one's first pairs
    int block = -1, ch_loaded = -1, cn = 0;
    int left_block = -1;  // SIGNAL: a block this CTA has left and not yet announced
    int ch = first_chunk + mine.x / t.nslabs, slab = mine.x % t.nslabs;
    for (int u = mine.x; u < mine.y; u += SIGNAL ? (int)gridDim.x : 1) {
        int c0 = 0;
        if (ch != ch_loaded) {
            const int4 chunk = t.chunks[ch];
            c0 = chunk.y;
            cn = chunk.z;
            if (SIGNAL && block >= 0 && chunk.x != block) {
                if (left_block >= 0) bucket_signal(t.sig, left_block);  // (only if a whole block went by within one unit)
                left_block = block;
            }
            block = chunk.x;
        }
        // the chunk's row lists, unless the unit before left them here: asynchronous copy into shared memory,
        // overlapped with the staging below
        if (ch != ch_loaded) {
            const int* start_in = t.csr_start + (size_t)ch * t.start_cap;
            const int4 head = __ldg(reinterpret_cast<const int4*>(start_in));
            for (int i = threadIdx.x; i < (head.y + 7) / 4; i += kBwdThreads) cp_async16(start + 4 * i, start_in + 4 * i);
            const uint16_t* ent_in = t.csr_ent + (size_t)ch * t.ent_cap;
            for (int i = threadIdx.x; i < (head.x + 7) / 8; i += kBwdThreads) cp_async16(ent + 8 * i, ent_in + 8 * i);
            for (int k = threadIdx.x; k < cn; k += kBwdThreads) {
                const int pair = __ldg(t.pairs + c0 + k).x;
                pairs_s[k] = pair;
                if (ONE) one_s[k] = make_int2(__float_as_int(a.dout[pair >> 1]), (2 * a.out_bucket[pair >> 1] + (pair & 1)) * x_row);
            }
            ch_loaded = ch;
            __syncthreads();  // the pair ids are in place
        }
        // stage this chunk's gradients at the feature-transformer pre-activation
        float4 sum_a = make_float4(0, 0, 0, 0), sum_b = sum_a;
        if (!fetched) fetch(warp * kPairsPerWarp + sub, cn, slab);
        for (int pl0 = warp * kPairsPerWarp + sub; pl0 < cn; pl0 += U * NW * kPairsPerWarp) {
#pragma unroll
            for (int k = 0; k < U; k++) {
                const int pl = pl0 + k * NW * kPairsPerWarp;
                if (pl >= cn) break;
                if (ONE) d[k] = scale4(d[k], __int_as_float(one_s[pl].x));
                float* out = g_s + pl * kTileCols + 4 * q;
                if (PAIRWISE) {
                    const float4 ga = make_float4((d[k].x * y1[k].x) * ft_act_bwd(1, y0[k].x), (d[k].y * y1[k].y) * ft_act_bwd(1, y0[k].y),
                                                  (d[k].z * y1[k].z) * ft_act_bwd(1, y0[k].z), (d[k].w * y1[k].w) * ft_act_bwd(1, y0[k].w));
                    const float4 gb = make_float4((d[k].x * y0[k].x) * ft_act_bwd(1, y1[k].x), (d[k].y * y0[k].y) * ft_act_bwd(1, y1[k].y),
                                                  (d[k].z * y0[k].z) * ft_act_bwd(1, y1[k].z), (d[k].w * y0[k].w) * ft_act_bwd(1, y1[k].w));
                    *reinterpret_cast<float4*>(out) = ga;
                    *reinterpret_cast<float4*>(out + 32) = gb;
                    sum_a = add4(sum_a, ga);
                    sum_b = add4(sum_b, gb);
                } else {
                    const float4 ga = make_float4(d[k].x * ft_act_bwd(a.act, y0[k].x), d[k].y * ft_act_bwd(a.act, y0[k].y),
                                                  d[k].z * ft_act_bwd(a.act, y0[k].z), d[k].w * ft_act_bwd(a.act, y0[k].w));
                    *reinterpret_cast<float4*>(out) = ga;
                    sum_a = add4(sum_a, ga);
                }
                if (pl + U * kStep < cn) fetch_one(k, pl + U * kStep, slab);
            }
        }
#pragma unroll
        for (int o = kLanes; o < 32; o <<= 1) {
            sum_a = add4(sum_a, make_float4(__shfl_xor_sync(0xffffffffu, sum_a.x, o), __shfl_xor_sync(0xffffffffu, sum_a.y, o),
                                            __shfl_xor_sync(0xffffffffu, sum_a.z, o), __shfl_xor_sync(0xffffffffu, sum_a.w, o)));
            if (PAIRWISE)
                sum_b = add4(sum_b, make_float4(__shfl_xor_sync(0xffffffffu, sum_b.x, o), __shfl_xor_sync(0xffffffffu, sum_b.y, o),
                                                __shfl_xor_sync(0xffffffffu, sum_b.z, o), __shfl_xor_sync(0xffffffffu, sum_b.w, o)));
        }
        if (sub == 0) {
            float* b = bias_s + warp * kTileCols + 4 * q;
            *reinterpret_cast<float4*>(b) = sum_a;
            if (PAIRWISE) *reinterpret_cast<float4*>(b + 32) = sum_b;
        }
        cp_async_wait_all();
        __syncthreads();
        if (SIGNAL && left_block >= 0) {
            bucket_signal(t.sig, left_block);
            left_block = -1;
        }
        // The next unit of a CTA that walks consecutive units is the same chunk's next slab: ask L2 for the lines
        // its staging will read (the neighbours of the ones just staged) now, so that they arrive during the walk.
        const bool next_slab = !SIGNAL && slab + 1 < t.nslabs && u + 1 < mine.y;
        if (next_slab && (int)threadIdx.x < cn) {
            const int pair = pairs_s[threadIdx.x], col = (slab + 1) * (PAIRWISE ? 32 : 64);
            if (PAIRWISE) {
                const float* pu = a.u + (size_t)pair * a.H + col;
                prefetch_l2(pu);
                prefetch_l2(pu + a.H / 2);
                if (!ONE) prefetch_l2(a.dx + (size_t)pair * x_row + col);
            } else {
                const size_t at = (size_t)pair * a.H + col;
                if (!ONE) prefetch_l2(a.dx + at);
                prefetch_l2(a.x + at);
                if (col + 32 < x_row) {
                    if (!ONE) prefetch_l2(a.dx + at + 32);
                    prefetch_l2(a.x + at + 32);
                }
            }
        }
        // The four table columns this lane sums.  Those past the width (the last slab of one that 64 does not divide) are not
        // the table's to write: their operands are zero, and zero sums are not written, but with ONE a loss gradient that is
        // not finite makes NaN of the zeros.  (Asked in the staging instead, or of every network: 2 to 4 % of the kernel.)
        const int col_w = !PAIRWISE ? slab * 64 + 4 * l16 : l16 < 8 ? slab * 32 + 4 * l16 : a.H / 2 + slab * 32 + 4 * (l16 - 8);
        const bool col_on = !ONE || (PAIRWISE ? slab * 32 + 4 * (l16 & 7) : col_w) < x_row;
        float* g_block = a.g_table + (size_t)block * R * a.H + col_w;
        if (threadIdx.x >= kBwdThreads - kTileCols) {
            const int j = (int)threadIdx.x - (kBwdThreads - kTileCols);
            float sum = 0.f;
#pragma unroll 8
            for (int w = 0; w < NW; w++) sum += bias_s[w * kTileCols + j];
            const bool on = !ONE || (PAIRWISE ? slab * 32 + (j & 31) : slab * 64 + j) < x_row;
            if (on && sum != 0.f) atomicAdd(a.g_bias + (!PAIRWISE ? slab * 64 + j : j < 32 ? slab * 32 + j : a.H / 2 + slab * 32 + j - 32), sum);
        }
        const int pieces = start[1];
        auto walk = [&](unsigned piece) {
            const f32x4 acc = sum_lines_even<!PAIRWISE>(smem_raw, reinterpret_cast<const uint2*>(ent) + (piece >> 17), (int)(piece >> 10) & 0x7f, lane16);
            const float4 g = make_float4(lo2(acc.a), hi2(acc.a), lo2(acc.b), hi2(acc.b));
            if (col_on && (g.x != 0.f || g.y != 0.f || g.z != 0.f || g.w != 0.f))
                atomicAdd(reinterpret_cast<float4*>(g_block + (size_t)(piece & 0x3ffu) * a.H), g);
        };
        // The pieces are dealt to the half warps to and fro, longest first, so that each gets the same mixture of lengths: whole rounds, which all
        // lanes of a warp walk together, then the shortest.  (A counter for the last quarter balanced no better, and its second copy of
        // the walk and the registers around it cost 1900 against 1844 us at 131072 positions x 2048 columns.)
        constexpr int HW = 2 * NW;
        const int h = 2 * warp + half, dealt = pieces / HW;
        unsigned piece = dealt > 0 ? (unsigned)start[4 + h] : 0u;
        for (int r = 0; r < dealt; r++) {
            const unsigned now = piece;
            if (r + 1 < dealt) piece = (unsigned)start[4 + (r + 1) * HW + (r & 1 ? h : HW - 1 - h)];
            walk(now);
        }
        __syncwarp();
        const int last = dealt * HW + h;
        if (last < pieces) walk((unsigned)start[4 + last]);
        fetched = next_slab;
        if (next_slab) fetch(warp * kPairsPerWarp + sub, cn, slab + 1);  // (arrives while the slowest warps finish)
        if (SIGNAL) {
            ch = first_chunk + (u + (int)gridDim.x) / t.nslabs;
            slab = (u + (int)gridDim.x) % t.nslabs;
        } else if (++slab == t.nslabs) {
            slab = 0;
            ch++;
        }
        __syncthreads();
    }
    if (SIGNAL && left_block >= 0) bucket_signal(t.sig, left_block);
    if (SIGNAL && block >= 0) bucket_signal(t.sig, block);
}

// ------------------------------------------------------- factoriser helper kernels
// table[i] = l0w[i] + l0f[i mod block]   (model/builder.rs:421-424 `repeat`, then `+`)
static __global__ void factoriser_merge_kernel(const float4* __restrict__ l0w, const float4* __restrict__ l0f,
                                        float4* __restrict__ table, size_t n4, size_t block4) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n4; i += (size_t)gridDim.x * blockDim.x)
        table[i] = add4(l0w[i], l0f[i % block4]);
}
// g_l0f[i] = sum over the tiled copies of g_l0w, first copy first (reduce.rs:96-120)
// `g_l0w` points at the first of `copies` consecutive copies; with `accumulate` the sum is added
// to what g_l0f already holds (the copies are then visited in several launches).
static __global__ void factoriser_grad_kernel(const float4* __restrict__ g_l0w, float4* __restrict__ g_l0f, size_t block4,
                                       int copies, int accumulate) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < block4; i += (size_t)gridDim.x * blockDim.x) {
        float4 acc = g_l0w[i];
        for (int k = 1; k < copies; k++) acc = add4(acc, g_l0w[(size_t)k * block4 + i]);
        g_l0f[i] = accumulate ? add4(g_l0f[i], acc) : acc;
    }
}

}  // namespace b200
