// Grouping of a batch on the device: the (position, perspective) pairs by table row block, with their prepared row lists,
// and the positions by output bucket, with every table that the step's kernels are cut by.  Nothing is read back: the
// host sizes the launches from the batch size alone (a tile or chunk that is not needed has count 0).
//
//   pass 1  one kernel per source (group_lists_kernel here, prep_featurise_kernel for raw records): per pair its block and
//           list length, per CTA of kGroupPositions positions a histogram of blocks and output buckets
//   pass 2  group_place_kernel: one CTA per window of kWindowPositions positions.  It sums the histograms before it (the
//           whole table of them is a few tens of KB; a long one has been summed up by group_scan_kernel), orders its pairs by
//           (block, list length) and writes their lists in place; CTA 0 also derives the tables.
//
// Pairs of one block and window lie in the order of their list lengths, so that neighbours, which the row walks serve two
// at a time, have lists of nearly the same length; a window is small enough that every stretch of a block's pairs holds
// the same mixture of lengths, which is what lets the walks cut the work by pair count.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels_ft.cuh"

namespace b200 {

constexpr int kGroupPositions = 128;   // positions per CTA of pass 1
constexpr int kWindowPositions = 512;  // positions per CTA of pass 2
constexpr int kGroupMaxBlocks = 256;   // most row blocks that the windows order; beyond, see group_many_* below
constexpr int kGroupMaxBuckets = 64;
constexpr int kDenseTile = 32;         // positions of one output bucket handled by one CTA of the dense kernels

struct GroupArgs {
    const uint16_t* stm;
    const uint16_t* nstm;  // [n][nnz] packed lists, 0xFFFF = empty
    const int* buckets;    // [n] output bucket per position (n_out_buckets > 1)
    int n, nnz, n_inputs, block_rows, nblocks, n_out_buckets;
    int* info;             // scratch [2n]: block << 8 | list length
    int* hist;             // scratch [CTAs of pass 1 + 1][nblocks + n_out_buckets]
    int* status;           // device or pinned host word
    int clear_status;      // pass 1 clears it first
    // pass 2
    int want_lists;        // pairs and lists are wanted (else only the positions' order and the dense tiles)
    int2* pairs;           // [2n] (pair id, list length), grouped by block
    uint16_t* lists;       // [2n][list_len] rows local to the block, in slot order, padded to 16 bytes with the zero row
    int list_len;
    int* order;            // [n] positions grouped by output bucket, or null
    int* block_begin;      // [nblocks + 1]
    int2* tiles;           // [max_tiles] dense tiles, or null
    int max_tiles;
    int4* chunks;          // [max_chunks] chunks of the tiled backward, or null
    int* chunk_begin;      // [nblocks + 1]
    int max_chunks, chunk_len;
    int* expect;           // [nblocks] CTAs of a whole-batch backward launch of `expect_grid` CTAs that work on each block
    int expect_grid, nslabs;
};

__host__ __device__ inline int group_ctas(int n) { return (n + kGroupPositions - 1) / kGroupPositions; }
__host__ __device__ inline int group_windows(int n) { return (n + kWindowPositions - 1) / kWindowPositions; }

// Every window reads all histograms, so that the reads grow with the square of the batch.  Up to 131072 positions that is the
// cheaper way (18 MB out of L2 with 17 bins, about 4 us, as much as one more launch); beyond, their running sums are formed once.
// Operator of 64 columns, 32 slots, 16 blocks, without and with the sums: 207 and 170 us at 262144 positions, 11.9 and 2.1 ms at
// 4 million.
inline bool group_scans(int n) { return group_ctas(n) > 1024; }

// hist[c][bin] -> sum of the rows before c, and the total in one more row.  grid = bins, block = 1024.
static __global__ void __launch_bounds__(1024) group_scan_kernel(int* hist, int ctas, int nbins) {
    step_begin(nullptr);
    __shared__ int warp_tot[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int* column = hist + blockIdx.x;
    int run = 0;
    for (int base = 0; base < ctas; base += 1024) {
        const int c = base + (int)threadIdx.x;
        const int own = c < ctas ? column[(size_t)c * nbins] : 0;
        int incl = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        if (lane == 31) warp_tot[warp] = incl;
        __syncthreads();
        const int before = __reduce_add_sync(0xffffffffu, lane < warp ? warp_tot[lane] : 0), all = __reduce_add_sync(0xffffffffu, warp_tot[lane]);
        if (c < ctas) column[(size_t)c * nbins] = run + before + incl - own;
        run += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) column[(size_t)ctas * nbins] = run;
}

// Whether a thread can take eight slots of a list with one load: the lists start on 16 bytes and hold 8, 16, 32 or 64 slots.
inline bool group_vec(const GroupArgs& g) {
    return (g.nnz == 8 || g.nnz == 16 || g.nnz == 32 || g.nnz == 64) && !(((uintptr_t)g.stm | (uintptr_t)g.nstm) & 15);
}
// eight slots: which of them hold a feature of the table
__device__ __forceinline__ int valid_slots(uint4 w, int n_inputs) {
    const uint32_t in[4] = {w.x, w.y, w.z, w.w};
    int m = 0;
#pragma unroll
    for (int h = 0; h < 4; h++) m |= ((in[h] & 0xffffu) < (uint32_t)n_inputs ? 1 : 0) << (2 * h) | ((in[h] >> 16) < (uint32_t)n_inputs ? 1 : 0) << (2 * h + 1);
    return m;
}

// Pass 1 from packed lists: with `vec` (group_vec) nnz / 8 threads per pair, else one warp per pair and eight pairs in
// flight; either way one round of loads per thread for lists of up to 32 slots.  grid = group_ctas(n), block = kGroupThreads.
constexpr int kGroupThreads = 1024;
static __global__ void __launch_bounds__(kGroupThreads) group_lists_kernel(GroupArgs g, int vec) {
    step_begin(nullptr);
    __shared__ int hist[kGroupMaxBlocks + kGroupMaxBuckets];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nbins = g.nblocks + g.n_out_buckets;
    for (int k = threadIdx.x; k < nbins; k += kGroupThreads) hist[k] = 0;
    if (blockIdx.x == 0 && threadIdx.x == 0 && g.clear_status) *g.status = 0;
    __syncthreads();
    const int first = 2 * kGroupPositions * (int)blockIdx.x, last = min(2 * g.n, first + 2 * kGroupPositions);
    // the block of a pair is the block of its first valid feature; a pair without any may go anywhere
    if (g.want_lists && vec) {
        const int q_of = g.nnz >> 3, shift = __ffs(q_of) - 1;
        for (int e = threadIdx.x; e < 2 * kGroupPositions << shift; e += kGroupThreads) {
            const int pair = first + (e >> shift), q = e & (q_of - 1);
            uint4 w = make_uint4(~0u, ~0u, ~0u, ~0u);
            if (pair < last) w = __ldg(reinterpret_cast<const uint4*>(((pair & 1) ? g.nstm : g.stm) + (size_t)(pair >> 1) * g.nnz) + q);
            const int m = valid_slots(w, g.n_inputs), at = __ffs(m) - 1;
            const uint32_t word = at < 2 ? w.x : at < 4 ? w.y : at < 6 ? w.z : w.w;
            // (place of the first feature, the feature): the smallest over the pair's threads
            unsigned best = m ? (unsigned)(8 * q + at) << 16 | (at & 1 ? word >> 16 : word & 0xffffu) : ~0u;
            int len = __popc(m);
            for (int o = 1; o < q_of; o <<= 1) {
                best = min(best, __shfl_xor_sync(0xffffffffu, best, o));
                len += __shfl_xor_sync(0xffffffffu, len, o);
            }
            if (q == 0 && pair < last) {
                const int block = len ? (int)(best & 0xffffu) / g.block_rows : 0;
                g.info[pair] = block << 8 | len;
                atomicAdd(&hist[block], 1);
            }
        }
    } else if (g.want_lists) {
        constexpr int U = 2 * kGroupPositions / (kGroupThreads / 32);
        uint32_t s0[U], s1[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int pair = first + U * warp + u;
            s0[u] = s1[u] = kNoFeature;
            if (pair < last) load_slots(((pair & 1) ? g.nstm : g.stm) + (size_t)(pair >> 1) * g.nnz, g.nnz, lane, s0[u], s1[u]);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int pair = first + U * warp + u;
            if (pair >= last) break;
            const unsigned m0 = __ballot_sync(0xffffffffu, s0[u] < (uint32_t)g.n_inputs);
            const unsigned m1 = __ballot_sync(0xffffffffu, s1[u] < (uint32_t)g.n_inputs);
            const uint32_t f = __shfl_sync(0xffffffffu, m0 ? s0[u] : s1[u], m0 ? __ffs(m0) - 1 : m1 ? __ffs(m1) - 1 : 0);
            if (lane == 0) {
                const int block = m0 | m1 ? (int)f / g.block_rows : 0;
                g.info[pair] = block << 8 | (__popc(m0) + __popc(m1));
                atomicAdd(&hist[block], 1);
            }
        }
    }
    if (g.n_out_buckets > 1)
        for (int i = first / 2 + threadIdx.x; i < last / 2; i += kGroupThreads) atomicAdd(&hist[g.nblocks + g.buckets[i]], 1);
    __syncthreads();
    for (int k = threadIdx.x; k < nbins; k += kGroupThreads) g.hist[(size_t)blockIdx.x * nbins + k] = hist[k];
}

// Exclusive sums of v[0 .. count) in place, v[count] = total.  One warp.
__device__ __forceinline__ void warp_exclusive_scan(int* v, int count, int lane) {
    int run = 0;
    for (int base = 0; base < count; base += 32) {
        const int own = base + lane < count ? v[base + lane] : 0;
        int incl = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        if (base + lane < count) v[base + lane] = run + incl - own;
        run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) v[count] = run;
}

// The tables that follow from the totals.  `block_at` [nblocks + 1] and `bucket_at` [n_out_buckets + 1] hold the first pair
// of every block and the first position of every bucket; `scan_s` [kGroupMaxBlocks + 1] is scratch.  All threads of a CTA.
__device__ inline void derive_tables(const GroupArgs& g, const int* block_at, const int* bucket_at, int* scan_s) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nb = g.nblocks;
    if (g.tiles && g.n_out_buckets > 1) {  // runs of up to kDenseTile positions of one bucket
        __syncthreads();
        for (int k = threadIdx.x; k < g.n_out_buckets; k += blockDim.x) scan_s[k] = (bucket_at[k + 1] - bucket_at[k] + kDenseTile - 1) / kDenseTile;
        __syncthreads();
        if (warp == 0) warp_exclusive_scan(scan_s, g.n_out_buckets, lane);
        __syncthreads();
        for (int i = threadIdx.x; i < g.max_tiles; i += blockDim.x) {
            int2 t = make_int2(0, 0);
            if (i < scan_s[g.n_out_buckets]) {
                int k = 0;
                while (i >= scan_s[k + 1]) k++;
                t.x = bucket_at[k] + kDenseTile * (i - scan_s[k]);
                t.y = min(kDenseTile, bucket_at[k + 1] - t.x);
            }
            g.tiles[i] = t;
        }
    }
    if (!g.want_lists) return;
    for (int b = threadIdx.x; b <= nb; b += blockDim.x) g.block_begin[b] = block_at[b];
    if (!g.chunks) return;
    // every block cut into the fewest equal runs of at most chunk_len pairs
    __syncthreads();
    for (int b = threadIdx.x; b < nb; b += blockDim.x) {
        const int pieces = (block_at[b + 1] - block_at[b] + g.chunk_len - 1) / g.chunk_len;
        const int size = pieces ? (block_at[b + 1] - block_at[b] + pieces - 1) / pieces : 1;
        scan_s[b] = (block_at[b + 1] - block_at[b] + size - 1) / size;
    }
    __syncthreads();
    if (warp == 0) warp_exclusive_scan(scan_s, nb, lane);
    __syncthreads();
    for (int b = threadIdx.x; b <= nb; b += blockDim.x) {
        g.chunk_begin[b] = scan_s[b];
        // a launch that announces finished blocks hands its CTAs the units k, k + grid, ... in block order
        if (b < nb && g.expect) g.expect[b] = min(g.expect_grid, g.nslabs * (scan_s[b + 1] - scan_s[b]));
    }
    for (int i = threadIdx.x; i < g.max_chunks; i += blockDim.x) {
        int4 c = make_int4(0, 0, 0, 0);
        if (i < scan_s[nb]) {
            int lo = 0, hi = nb;  // the last block whose first chunk is not past i
            while (hi - lo > 1) {
                const int mid = (lo + hi) / 2;
                (scan_s[mid] <= i ? lo : hi) = mid;
            }
            const int pairs = block_at[lo + 1] - block_at[lo], pieces = (pairs + g.chunk_len - 1) / g.chunk_len;
            const int size = (pairs + pieces - 1) / pieces, at = block_at[lo] + size * (i - scan_s[lo]);
            c = make_int4(lo, at, min(size, block_at[lo + 1] - at), 0);
        }
        g.chunks[i] = c;
    }
}

// One pair's prepared list by a whole warp: the valid rows inside the pair's block, compacted in slot order, the last
// 16-byte group filled with the zero row.  Any list length and alignment.  Returns the number of rows.
// (s0, s1: this lane's slots of the pair.)
__device__ __forceinline__ int prepare_list_warp(const GroupArgs& g, uint32_t s0, uint32_t s1, int block, uint16_t* list, int lane) {
    const bool v0 = s0 < (uint32_t)g.n_inputs, v1 = s1 < (uint32_t)g.n_inputs;
    const int row0 = (int)s0 - block * g.block_rows, row1 = (int)s1 - block * g.block_rows;
    const bool in0 = v0 && (unsigned)row0 < (unsigned)g.block_rows, in1 = v1 && (unsigned)row1 < (unsigned)g.block_rows;
    if ((v0 && !in0) || (v1 && !in1)) *g.status = kStatusOutsideBlock;  // dropped, and reported
    const unsigned m0 = __ballot_sync(0xffffffffu, in0), m1 = __ballot_sync(0xffffffffu, in1);
    const unsigned lt = (1u << lane) - 1u;
    const int cnt0 = __popc(m0), cnt = cnt0 + __popc(m1), cnt8 = (cnt + 7) & ~7;
    if (in0) list[__popc(m0 & lt)] = (uint16_t)row0;
    if (in1) list[cnt0 + __popc(m1 & lt)] = (uint16_t)row1;
    if (lane < cnt8 - cnt) list[cnt + lane] = (uint16_t)g.block_rows;
    return cnt;
}

constexpr int kPlaceThreads = 2 * kWindowPositions;
constexpr int kCountedBlocks = 32;  // up to as many row blocks a window orders its pairs by counting, beyond by sorting

// Pass 2.  grid = group_windows(n) CTAs of one thread per pair of the window.  `vec`: see group_vec; `scanned`: the histograms are
// running sums already (group_scan_kernel).
// Latency bound (one CTA per SM at most for ordinary batches): one sweep over the histograms, a counting sort (a bitonic one
// for many blocks: its 45 barriers took a third of the kernel's 13 us), one gather of the lists.
static __global__ void __launch_bounds__(kPlaceThreads) group_place_kernel(GroupArgs g, int vec, int scanned) {
    step_begin(nullptr);
    __shared__ int before[kGroupMaxBlocks + kGroupMaxBuckets], block_at[kGroupMaxBlocks + 1], bucket_at[kGroupMaxBuckets + 1];
    __shared__ int scan_s[kGroupMaxBlocks + 1], run_start[kGroupMaxBlocks];
    __shared__ unsigned key_s[kPlaceThreads];
    __shared__ int counter_s[kCountedBlocks * 65];
    __shared__ int place_s[kPlaceThreads], warp_count[kWindowPositions / 32][kGroupMaxBuckets];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tid = threadIdx.x;
    const int nb = g.nblocks, nbins = nb + g.n_out_buckets;
    for (int k = tid; k < nbins; k += kPlaceThreads) before[k] = 0;
    for (int k = tid; k <= kGroupMaxBlocks; k += kPlaceThreads) block_at[k] = 0;
    if (tid <= kGroupMaxBuckets) bucket_at[tid] = 0;
    __syncthreads();
    if (scanned) {
        const int ctas = group_ctas(g.n), mine = (int)blockIdx.x * (kWindowPositions / kGroupPositions);
        if (tid < nbins) {
            before[tid] = __ldcg(g.hist + (size_t)mine * nbins + tid);
            *(tid < nb ? &block_at[tid] : &bucket_at[tid - nb]) = __ldcg(g.hist + (size_t)ctas * nbins + tid);
        }
    } else {  // totals, and what lies before this window, of every bin
        int width = 1;
        while (width < nbins) width <<= 1;
        const int bin = tid & (width - 1), ctas = group_ctas(g.n), mine = (int)blockIdx.x * (kWindowPositions / kGroupPositions);
        int total = 0, prior = 0;
        if (bin < nbins) {
            for (int c = tid / width; c < ctas; c += kPlaceThreads / width) {
                const int v = __ldcg(g.hist + (size_t)c * nbins + bin);
                total += v;
                if (c < mine) prior += v;
            }
            if (total) atomicAdd(bin < nb ? &block_at[bin] : &bucket_at[bin - nb], total);
            if (prior) atomicAdd(&before[bin], prior);
        }
    }
    __syncthreads();
    if (warp == 0) warp_exclusive_scan(block_at, nb, lane);
    if (warp == 1) warp_exclusive_scan(bucket_at, g.n_out_buckets, lane);
    const int base = (int)blockIdx.x * kPlaceThreads;  // first pair of the window
    const int live = min(kPlaceThreads, 2 * g.n - base);
    if (g.want_lists) {
        unsigned key = 0xffffffffu;
        if (tid < live) {
            const unsigned info = (unsigned)g.info[base + tid];
            key = (info >> 8) << 17 | (info & 0x7fu) << 10 | (unsigned)tid;
        }
        if (nb <= kCountedBlocks) {
            // one counter per block and length; pairs of the same block and length come in any order
            constexpr int kLengths = 65, B = (kCountedBlocks * kLengths + kPlaceThreads - 1) / kPlaceThreads;
            const int bins = nb * kLengths;
            for (int k = tid; k < bins; k += kPlaceThreads) counter_s[k] = 0;
            __syncthreads();
            const int bin = (int)(key >> 17) * kLengths + (int)(key >> 10 & 0x7fu);
            int rank = 0;
            if (tid < live) rank = atomicAdd(&counter_s[bin], 1);
            __syncthreads();
            int own[B], sum = 0;
#pragma unroll
            for (int k = 0; k < B; k++) {
                own[k] = tid * B + k < bins ? counter_s[tid * B + k] : 0;
                sum += own[k];
            }
            int incl = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += up;
            }
            if (lane == 31) place_s[warp] = incl;
            __syncthreads();
            int at = incl - sum + __reduce_add_sync(0xffffffffu, lane < warp ? place_s[lane] : 0);
#pragma unroll
            for (int k = 0; k < B; k++) {
                if (tid * B + k < bins) counter_s[tid * B + k] = at;
                at += own[k];
            }
            __syncthreads();
            if (tid < nb) run_start[tid] = counter_s[tid * kLengths];
            if (tid < live) key_s[counter_s[bin] + rank] = key;
            __syncthreads();
            key = key_s[tid];
        } else {
            for (int k = 2; k <= kPlaceThreads; k <<= 1)
                for (int j = k >> 1; j > 0; j >>= 1) {
                    unsigned other;
                    if (j >= 32) {
                        __syncthreads();
                        key_s[tid] = key;
                        __syncthreads();
                        other = key_s[tid ^ j];
                    } else {
                        other = __shfl_xor_sync(0xffffffffu, key, j);
                    }
                    const bool keep_min = ((tid & j) == 0) == ((tid & k) == 0);
                    key = keep_min ? min(key, other) : max(key, other);
                }
            __syncthreads();
            key_s[tid] = key;
            __syncthreads();
            if (tid < live && (tid == 0 || (key_s[tid - 1] >> 17) != (key >> 17))) run_start[key >> 17] = tid;
            __syncthreads();
        }
        if (tid < live) place_s[tid] = block_at[key >> 17] + before[key >> 17] + tid - run_start[key >> 17];
        __syncthreads();
        if (vec) {
            const int q_of = g.nnz >> 3, shift = __ffs(q_of) - 1;  // threads per pair
            constexpr int U = 4;                                   // loads in flight
            for (int e0 = tid; e0 < kPlaceThreads << shift; e0 += U * kPlaceThreads) {
                uint4 w[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int e = e0 + u * kPlaceThreads, j = e >> shift;
                    w[u] = make_uint4(~0u, ~0u, ~0u, ~0u);
                    if (j < live) {
                        const int pair = base + (int)(key_s[j] & 0x3ffu);
                        w[u] = __ldcg(reinterpret_cast<const uint4*>(((pair & 1) ? g.nstm : g.stm) + (size_t)(pair >> 1) * g.nnz) + (e & (q_of - 1)));
                    }
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int e = e0 + u * kPlaceThreads, j = e >> shift, q = e & (q_of - 1);
                    const bool on = j < live;
                    const unsigned k = on ? key_s[j] : 0u;
                    const int pair = base + (int)(k & 0x3ffu), len = (int)(k >> 10) & 0x7f;
                    const uint32_t row0 = (k >> 17) * (uint32_t)g.block_rows;
                    const int expect = on ? (1 << max(0, min(8, len - 8 * q))) - 1 : 0;
                    const uint32_t in[4] = {w[u].x, w[u].y, w[u].z, w[u].w};
                    uint32_t out[4];
                    int inside = 0;
#pragma unroll
                    for (int h = 0; h < 4; h++) {
                        const uint32_t a = in[h] & 0xffffu, b = in[h] >> 16, ra = a - row0, rb = b - row0;
                        const bool ina = a < (uint32_t)g.n_inputs && ra < (uint32_t)g.block_rows, inb = b < (uint32_t)g.n_inputs && rb < (uint32_t)g.block_rows;
                        inside |= (ina ? 1 : 0) << (2 * h) | (inb ? 1 : 0) << (2 * h + 1);
                        out[h] = (ina ? ra : (uint32_t)g.block_rows) | (inb ? rb : (uint32_t)g.block_rows) << 16;
                    }
                    // the usual list: its `len` features fill the first slots and lie in the block
                    const unsigned odd = __ballot_sync(0xffffffffu, inside != expect);
                    const unsigned group = ((1u << q_of) - 1u) << (lane & ~(q_of - 1));
                    if (!on) continue;
                    uint16_t* list = g.lists + (size_t)place_s[j] * g.list_len;
                    if (!(odd & group)) {
                        *reinterpret_cast<uint4*>(list + 8 * q) = make_uint4(out[0], out[1], out[2], out[3]);
                        if (q == 0) g.pairs[place_s[j]] = make_int2(pair, len);
                    } else if (q == 0) {  // holes or features outside the block: one thread compacts the list
                        const uint16_t* src = ((pair & 1) ? g.nstm : g.stm) + (size_t)(pair >> 1) * g.nnz;
                        int cnt = 0;
                        for (int s = 0; s < g.nnz; s++) {
                            const uint32_t f = src[s], row = f - row0;
                            if (f >= (uint32_t)g.n_inputs) continue;
                            if (row < (uint32_t)g.block_rows) list[cnt++] = (uint16_t)row;
                            else *g.status = kStatusOutsideBlock;  // dropped, and reported (the one bit there is)
                        }
                        g.pairs[place_s[j]] = make_int2(pair, cnt);
                        for (; cnt & 7; cnt++) list[cnt] = (uint16_t)g.block_rows;
                    }
                }
            }
        } else {
            constexpr int U = 8, NW = kPlaceThreads / 32;
            for (int j0 = warp; j0 < live; j0 += U * NW) {
                uint32_t s0[U], s1[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int j = j0 + u * NW, pair = base + (int)(key_s[min(j, live - 1)] & 0x3ffu);
                    load_slots(((pair & 1) ? g.nstm : g.stm) + (size_t)(pair >> 1) * g.nnz, g.nnz, lane, s0[u], s1[u]);
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int j = j0 + u * NW;
                    if (j >= live) break;
                    const unsigned k = key_s[j];
                    const int cnt = prepare_list_warp(g, s0[u], s1[u], (int)(k >> 17), g.lists + (size_t)place_s[j] * g.list_len, lane);
                    if (lane == 0) g.pairs[place_s[j]] = make_int2(base + (int)(k & 0x3ffu), cnt);
                }
            }
        }
    }
    if (g.order) {  // positions by output bucket, in ascending order inside a bucket
        __syncthreads();
        for (int k = tid; k < (kWindowPositions / 32) * kGroupMaxBuckets; k += kPlaceThreads) (&warp_count[0][0])[k] = 0;
        __syncthreads();
        const int id = (int)blockIdx.x * kWindowPositions + tid;
        const bool on = tid < kWindowPositions && id < g.n;
        const int bucket = on ? g.buckets[id] : g.n_out_buckets;  // the others share a key of their own
        const unsigned same = __match_any_sync(0xffffffffu, bucket);
        const int rank = __popc(same & ((1u << lane) - 1u));
        if (on && rank == 0) warp_count[warp][bucket] = __popc(same);
        __syncthreads();
        if (on) {
            int at = bucket_at[bucket] + before[nb + bucket] + rank;
            for (int w = 0; w < warp; w++) at += warp_count[w][bucket];
            g.order[at] = id;
        }
    }
    if (blockIdx.x == 0) derive_tables(g, block_at, bucket_at, scan_s);
}

// More row blocks than a window's tables hold: counts and places through global counters (`count` [nblocks +
// n_out_buckets], zero on entry), in no particular order inside a block.
static __global__ void __launch_bounds__(256) group_many_count_kernel(GroupArgs g, int* count) {
    const int lane = threadIdx.x & 31, pair = (int)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (blockIdx.x == 0 && threadIdx.x == 0 && g.clear_status) *g.status = 0;
    if (pair >= 2 * g.n) return;
    uint32_t s0, s1;
    load_slots(((pair & 1) ? g.nstm : g.stm) + (size_t)(pair >> 1) * g.nnz, g.nnz, lane, s0, s1);
    const unsigned m0 = __ballot_sync(0xffffffffu, s0 < (uint32_t)g.n_inputs), m1 = __ballot_sync(0xffffffffu, s1 < (uint32_t)g.n_inputs);
    const uint32_t f = __shfl_sync(0xffffffffu, m0 ? s0 : s1, m0 ? __ffs(m0) - 1 : m1 ? __ffs(m1) - 1 : 0);
    if (lane == 0) {
        const int block = m0 | m1 ? (int)f / g.block_rows : 0;
        g.info[pair] = block;
        if (g.want_lists) atomicAdd(count + block, 1);
        if (g.n_out_buckets > 1 && !(pair & 1)) atomicAdd(count + g.nblocks + g.buckets[pair >> 1], 1);
    }
}
// One CTA: `at` [nblocks + n_out_buckets + 2] and `scratch` [max(nblocks, n_out_buckets) + 1] in global memory; `count` becomes the cursors.
static __global__ void __launch_bounds__(1024) group_many_scan_kernel(GroupArgs g, int* count, int* at, int* scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nb = g.nblocks;
    int* bucket_at = at + nb + 1;
    for (int k = threadIdx.x; k < nb; k += blockDim.x) at[k] = count[k];
    for (int k = threadIdx.x; k < g.n_out_buckets; k += blockDim.x) bucket_at[k] = count[nb + k];
    __syncthreads();
    if (warp == 0) warp_exclusive_scan(at, nb, lane);
    if (warp == 1) warp_exclusive_scan(bucket_at, g.n_out_buckets, lane);
    __syncthreads();
    for (int k = threadIdx.x; k < nb; k += blockDim.x) count[k] = at[k];
    for (int k = threadIdx.x; k < g.n_out_buckets; k += blockDim.x) count[nb + k] = bucket_at[k];
    derive_tables(g, at, bucket_at, scratch);
}
static __global__ void __launch_bounds__(256) group_many_place_kernel(GroupArgs g, int* cursor) {
    const int lane = threadIdx.x & 31, pair = (int)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (pair >= 2 * g.n) return;
    if (g.want_lists) {
        const int block = g.info[pair];
        int place = 0;
        if (lane == 0) place = atomicAdd(cursor + block, 1);
        place = __shfl_sync(0xffffffffu, place, 0);
        uint32_t s0, s1;
        load_slots(((pair & 1) ? g.nstm : g.stm) + (size_t)(pair >> 1) * g.nnz, g.nnz, lane, s0, s1);
        const int cnt = prepare_list_warp(g, s0, s1, block, g.lists + (size_t)place * g.list_len, lane);
        if (lane == 0) g.pairs[place] = make_int2(pair, cnt);
    }
    if (g.order && lane == 0 && !(pair & 1)) g.order[atomicAdd(cursor + g.nblocks + g.buckets[pair >> 1], 1)] = pair >> 1;
}

}  // namespace b200
