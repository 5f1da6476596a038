// Batch preparation on the device, from raw 32-byte position records: the featurisers, the output
// bucket and the target blend, and the first pass of the grouping (kernels_group.cuh).
//
// Reference semantics (jw1912/bullet): Chess768::map_features
// crates/bullet_lib/src/game/inputs/chess768.rs:20-30, ChessBucketsMirrored
// crates/bullet_lib/src/game/inputs/chess_buckets.rs:57-88, Ataxx147
// crates/bullet_lib/src/game/inputs/ataxx147.rs:18-27, MaterialCount
// crates/bullet_lib/src/game/outputs.rs:24-31, the mapper's layout and target blend
// crates/bullet_lib/src/value.rs:77-117; record layouts as restated in examples/tests/test4.rs:8-36
// and examples/ataxx.rs:8-18.  The host mappers (host_map.h) are the same functions; a GPU test holds
// the two against each other bit for bit.  The host has checked the records: none holds more pieces than slots, and
// every one has an output bucket.
//
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels_group.cuh"

namespace b200 {

struct PrepArgs {
    const uint4* records;   // [n] raw records (32 bytes = two uint4 each)
    int game;
    const int* expanded;    // [64] 768 * king bucket of every square (king-bucketed chess inputs)
    const float* win_rate;  // [65536] sigmoid(score / scale) for every 16-bit score, index score + 32768
    const float* given;     // the targets as the host has formed them, or null
    float blend;
    uint16_t* stm;          // out [n][nnz], 0xFFFF = empty
    uint16_t* nstm;
    int* buckets;           // out [n]
    float* targets;         // out [n]
};

// game codes as in bullet_b200.h: 0 chess 768, 1 king-bucketed mirrored chess, 2 ataxx 147.
// One thread per position for what a position has one of (bucket, target), then one warp per position for the lists: a lane
// owns two squares, and the place of a piece in the list is the number of occupied squares below it, so nothing loops over
// pieces.  (A thread per position that walked its bitboards took 14 us for 16384 positions and stored two bytes at a time.)
// The records may lie in pinned host memory: they are read once, coalesced.  grid = group_ctas(n), block = kPrepThreads.
constexpr int kPrepThreads = 512;
static __global__ void __launch_bounds__(kPrepThreads) prep_featurise_kernel(PrepArgs p, GroupArgs g) {
    step_begin(nullptr);
    __shared__ uint4 record_s[kGroupPositions][2];
    __shared__ int hist[kGroupMaxBlocks + kGroupMaxBuckets];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nnz = g.nnz;
    // with more row blocks than the windows order, the pairs are counted by a kernel of their own
    const bool count_here = g.nblocks <= kGroupMaxBlocks;
    const int nbins = count_here ? g.nblocks + g.n_out_buckets : 0;
    const int first = (int)blockIdx.x * kGroupPositions, live = min(kGroupPositions, g.n - first);
    for (int k = threadIdx.x; k < nbins; k += kPrepThreads) hist[k] = 0;
    if (blockIdx.x == 0 && threadIdx.x == 0 && g.clear_status) *g.status = 0;
    static_assert(kPrepThreads >= 2 * kGroupPositions, "one 16-byte half of a record per thread");
    if ((int)threadIdx.x < 2 * live) record_s[threadIdx.x >> 1][threadIdx.x & 1] = p.records[2 * first + threadIdx.x];
    __syncthreads();
    if ((int)threadIdx.x < live) {
        const uint4 hi = record_s[threadIdx.x][1];
        // both record types keep score (i16) at byte 24 and the result at byte 26
        const int score = (int)(short)(hi.z & 0xffffu), result = (int)((hi.z >> 16) & 0xffu), i = first + (int)threadIdx.x;
        int bucket = 0;
        if (g.n_out_buckets > 1) {
            const uint4 lo = record_s[threadIdx.x][0];
            const int divisor = (32 + g.n_out_buckets - 1) / g.n_out_buckets;
            bucket = (__popc(lo.x) + __popc(lo.y) - 2) / divisor;
            if (count_here) atomicAdd(&hist[g.nblocks + bucket], 1);
        }
        p.buckets[i] = bucket;
        // blend * result / 2 + (1 - blend) * sigmoid(score / scale), every operation rounded on its own as the
        // host compiler does it (no fused multiply-add)
        if (p.given) {
            p.targets[i] = p.given[i];
        } else {
            const float wr = p.win_rate[score + 32768];
            p.targets[i] = __fadd_rn(__fmul_rn(p.blend, __fdiv_rn((float)result, 2.0f)), __fmul_rn(__fsub_rn(1.0f, p.blend), wr));
        }
    }
    const unsigned below = (1u << lane) - 1u;
#pragma unroll 4
    for (int r = warp; r < live; r += kPrepThreads / 32) {
        const uint4 lo = record_s[r][0], hi = record_s[r][1];
        uint16_t* s = p.stm + (size_t)(first + r) * nnz;
        uint16_t* t = p.nstm + (size_t)(first + r) * nnz;
        int count = 0, first_s = -1, first_t = -1, valid_s = 0, valid_t = 0;
        // 32 squares at a time: `on` says whether this lane's square has a piece, whose features are fs and ft
        auto put = [&](bool on, int fs, int ft) {
            const unsigned m = __ballot_sync(0xffffffffu, on);
            const bool in_s = on && (unsigned)fs < (unsigned)g.n_inputs, in_t = on && (unsigned)ft < (unsigned)g.n_inputs;
            const int at = count + __popc(m & below);
            if (on && at < nnz) {
                s[at] = in_s ? (uint16_t)fs : (uint16_t)kNoFeature;
                t[at] = in_t ? (uint16_t)ft : (uint16_t)kNoFeature;
            }
            const unsigned ms = __ballot_sync(0xffffffffu, in_s), mt = __ballot_sync(0xffffffffu, in_t);
            if (ms && first_s < 0) first_s = __shfl_sync(0xffffffffu, fs, __ffs(ms) - 1);
            if (mt && first_t < 0) first_t = __shfl_sync(0xffffffffu, ft, __ffs(mt) - 1);
            valid_s += __popc(ms);
            valid_t += __popc(mt);
            count += __popc(m);
        };
        if (p.game == 2) {  // own stones, their stones, blocked cells: the other side swaps the first two planes
            const unsigned words[6] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y};
#pragma unroll
            for (int plane = 0; plane < 3; plane++)
#pragma unroll
                for (int half = 0; half < 2; half++) {
                    const int sq = 32 * half + lane;
                    put((words[2 * plane + half] >> lane) & 1u, 49 * plane + sq, (plane == 0 ? 49 : plane == 1 ? 0 : 98) + sq);
                }
        } else {
            const unsigned occ[2] = {lo.x, lo.y};
            const int ksq = (int)((hi.z >> 24) & 0xffu), opp_ksq = (int)(hi.w & 0xffu);
            int us_base = 0, us_flip = 0, them_base = 0, them_flip = 0;
            if (p.game == 1) {
                us_base = __ldg(p.expanded + (ksq & 63));
                us_flip = (ksq & 7) > 3 ? 7 : 0;  // the king on files e..h mirrors the board
                them_base = __ldg(p.expanded + (opp_ksq & 63));
                them_flip = (opp_ksq & 7) > 3 ? 7 : 0;
            }
#pragma unroll
            for (int half = 0; half < 2; half++) {
                // 4-bit piece codes, two per byte, in ascending square order of the occupancy
                const int piece = (half ? __popc(occ[0]) : 0) + __popc(occ[half] & below);
                const unsigned word = piece & 16 ? (piece & 8 ? hi.y : hi.x) : (piece & 8 ? lo.w : lo.z);
                const int code = (int)(word >> ((piece & 7) * 4)) & 15, sq = 32 * half + lane;
                const int theirs = (code >> 3) & 1, type = code & 7;
                put((occ[half] >> lane) & 1u, us_base + ((384 * theirs + 64 * type + sq) ^ us_flip),
                    them_base + ((384 * (1 - theirs) + 64 * type + (sq ^ 56)) ^ them_flip));
            }
        }
        for (int k = count + lane; k < nnz; k += 32) s[k] = t[k] = (uint16_t)kNoFeature;
        if (count_here && lane == 0) {
            const int bs = first_s < 0 ? 0 : first_s / g.block_rows, bt = first_t < 0 ? 0 : first_t / g.block_rows;
            *reinterpret_cast<int2*>(g.info + 2 * (first + r)) = make_int2(bs << 8 | valid_s, bt << 8 | valid_t);
            if (g.want_lists) {
                atomicAdd(&hist[bs], 1);
                atomicAdd(&hist[bt], 1);
            }
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < nbins; k += kPrepThreads) g.hist[(size_t)blockIdx.x * nbins + k] = hist[k];
}

}  // namespace b200
