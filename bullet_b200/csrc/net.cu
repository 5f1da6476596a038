// b200_net: device state, staging slots and the fixed step schedule behind the C ABI.
//
// Replaces, for the NNUE training step only, what the reference assembles at run time from
// generated CUDA text: Function::new/prealloc/execute (crates/gpu/src/function.rs:73-280),
// the per-weight AdamW launches (crates/trainer/src/optimiser/adam.rs:217-291) and the
// batch copies of PreparedBatchHost (crates/trainer/src/run/dataloader.rs:41-61).  All
// device memory is allocated once in b200_net_create; a step only enqueues kernels.
//
// HBM layout
//   P, G, M, V   flat fp32 buffers: a 256-byte head whose first float (in G) is the summed
//                loss, then every tensor in name order (l0b, l0f, l1b, l1w, ...) except l0w,
//                which comes last; each tensor starts on a 256-byte boundary.  A
//                data-parallel host moves gradients and loss with one all-reduce of G, or
//                in parts: runs of l0w row blocks as the backward finishes them, then the
//                head (loss and all other tensors) in one piece.
//   table        l0w + tiled l0f (only with a factoriser; otherwise an alias of l0w in P)
//   x, u, dx     activations kept between forward and backward, position-major
//   slots        per staging slot one pinned host block and one device block holding the
//                packed u16 index lists, buckets, targets and the two visiting orders
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/bullet_b200.h"
#include "common.h"
#include "kernels_dense_mma.cuh"
#include "kernels_dense_one.cuh"
#include "kernels_ft.cuh"
#include "kernels_ft_mma.cuh"
#include "kernels_opt.cuh"
#include "kernels_prep.cuh"
#include "host_map.h"
#include "op_pool.h"

#define CK(call)                                                                                          \
    do {                                                                                                  \
        cudaError_t e_ = (call);                                                                          \
        if (e_ != cudaSuccess)                                                                            \
            return b200::fail(B200_ERR_CUDA, "%s failed: %s (%d) at %s:%d", #call, cudaGetErrorString(e_), \
                              (int)e_, __FILE__, __LINE__);                                               \
    } while (0)

// after every kernel launch: surface a launch error, count the launch
#define LAUNCHED(net)            \
    do {                         \
        CK(cudaGetLastError());  \
        (net)->launches++;       \
    } while (0)

namespace {

constexpr int64_t kAlignFloats = 64;       // 256-byte tensor alignment in the flat buffers
constexpr int kGatherRowsPerPosition = 34;  // active features of both perspectives of a middling chess position
constexpr long long kGatherMostBytes = 100 << 20, kGatherMostPerRow = 200 << 10;  // see b200_net::fwd_tiled
constexpr long long kGatherMore = 8 << 20;
constexpr int64_t kClearInForward = 2 << 20;  // floats of a gradient buffer that the forward kernel clears itself
constexpr int kDirectOutputs = 256;        // up to as many outputs of an evaluation the kernel stores to pinned memory itself
constexpr int kMinItemPairs = 128;         // a forward work item serves at least this many pairs per tile load

struct Tensor {
    std::string name;
    int64_t n = 0, off = 0;
    int64_t rows = 0, cols = 0;  // column-major shape, as the reference's Shape(rows, cols)
    b200_adamw_params hp{0.01f, 0.9f, 0.999f, -1.98f, 1.98f};
    // which update rule: AdamW, RAdam, or RAdam under Ranger's lookahead (crates/trainer/src/optimiser/{radam,ranger}.rs)
    int opt_kind = B200_OPT_ADAMW;
    float n_sma_threshold = 5.0f, alpha = 0.5f;
    int lookahead_k = 6;
};

struct Slot {
    char* d_blob = nullptr;
    char* h_blob = nullptr;
    int n = 0;
    int n_dtiles = 0;  // CTA tiles of the dense kernels: as many as there can be, the rest are empty
    bool wide = true;                 // shape of the tiled backward that its chunks were cut for
    bool mma = false;                 // ... or for ft_backward_mma_kernel
    int n_chunks = 0, chunk_len = 0;  // the same for the chunks of the tiled FT backward held in off_chunks, and their size
    int expect_grid = 0;              // grid size the per-block CTA counts in off_bexpect were made for
    // derived from the indices alone, so built once per upload on the copy stream (or on first use):
    uint16_t* lists = nullptr;        // prepared per-pair row lists of the tiled kernels
    uint16_t* csr_ent = nullptr;      // per-chunk row-major lists of the tiled backward
    int* csr_start = nullptr;
    bool prepared = false, csr_built = false;
    // what crosses PCIe comes first: either the packed lists, buckets, targets and (if the host made them) the dense
    // kernels' order and tiles, or the raw records; everything behind is written on the device
    size_t off_stm = 0, off_nstm = 0, off_buckets = 0, off_targets = 0, off_order = 0, off_dtiles = 0, off_records = 0, off_pairs = 0,
           off_blocks = 0, off_chunks = 0, off_cbegin = 0, off_bexpect = 0, off_status = 0, off_info = 0, off_hist = 0, bytes = 0;
    size_t off_many[3] = {0, 0, 0};   // counters of the grouping by more row blocks than its windows hold
    cudaEvent_t ready = nullptr, consumed = nullptr;
    bool has_ready = false, has_consumed = false;
    template <class T>
    T* dev(size_t off) const { return reinterpret_cast<T*>(d_blob + off); }
    template <class T>
    T* host(size_t off) const { return reinterpret_cast<T*>(h_blob + off); }
};

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

}  // namespace

struct b200_net {
    int device = 0;
    int sm_count = 1;  // cudaDevAttrMultiProcessorCount of `device`: grids are sized in waves of it
    cudaStream_t stream = nullptr, copy_stream = nullptr;
    // clears the gradient buffer beside the feature-transformer forward, which does not touch it
    cudaStream_t zero_stream = nullptr;
    cudaEvent_t zero_fork = nullptr, zero_done = nullptr;
    bool zero_pending = false;
    bool own_stream = false;
    b200_net_desc d{};
    std::vector<Tensor> tensors;
    int64_t n_flat = 0;
    float *P = nullptr, *G = nullptr, *M = nullptr, *V = nullptr, *table = nullptr;
    float *x = nullptr, *u = nullptr, *dx = nullptr, *a1 = nullptr, *a2 = nullptr, *out = nullptr, *w1g = nullptr;
    uint32_t* dz_frag = nullptr;     // the gradient at the first dense layer's pre-activation as an operand of its weight gradient
    float* dense_partial = nullptr;  // the first dense layer's sums of slices of its columns
    uint32_t *w1f = nullptr, *w1d = nullptr;  // the first dense layer's fragment tables (dense_mma)
    float* dz[3] = {nullptr, nullptr, nullptr};
    int wgrad_per_sm = 0;          // resident CTAs per SM of the first layer's weight-gradient kernel (looked up once)
    int status_slot = -1;          // slot whose status word the running step reports (-1: the step used no tiled kernel)
    // pinned read-back ring: loss and status word of the last kLossRing updates
    static constexpr int kLossRing = 4;
    int* h_status = nullptr;
    int* d_status = nullptr;       // [kLossRing] the slot's status word, saved before the slot is released to the uploader
    float* h_loss = nullptr;
    char* h_pinned = nullptr;      // the one pinned allocation that the slots' blocks, h_out and the ring lie in
    float* h_out = nullptr;        // pinned [max_batch]: network outputs of an evaluation
    cudaEvent_t loss_ev[kLossRing] = {};
    int64_t updates = 0;
    Slot slots[B200_NUM_SLOTS];
    int ft_fwd_mode = B200_FT_AUTO, ft_bwd_mode = B200_FT_AUTO;
    bool bwd_wide = true;  // shape of the tiled backward (see kChunkMost)
    int bwd_products = -1;  // small tables: the product of bytes instead of the walk over row lists, always (1), never (0) or where it pays
    int exchange_bulk = 0;  // the peer exchange moves gradients and weights with bulk asynchronous copies (measured no faster)
    int wide_chunk = 0;    // the largest chunk of the 1024-thread backward that fits into shared memory
    // Pairs per chunk for a batch of n positions: large chunks save reductions and list copies per pair, small ones fill the
    // SMs evenly when there are few units.  Measured, a unit takes a part that grows with the table's rows and the chunk's
    // pairs (clocks, 768 rows and 17 of 32 slots active: 13.4 k + 48 per pair; 147 rows, 27 of 49: 6.6 k + 78 per pair), and a
    // CTA takes whole units.
    int bwd_chunk(int n) const {
        if (!bwd_wide) return b200::ft_bwd_chunk_narrow(d.nnz);
        int best = wide_chunk;
        double least = 1e30;
        for (int len = wide_chunk; len >= b200::kChunkLeast; len -= 8) {
            const double chunks = nblocks > 1 ? 2.0 * n / len + 0.5 * nblocks : (double)((2LL * n + len - 1) / len);
            const double pairs = std::min<double>(len, 2.0 * n / chunks);
            const double units = chunks * nslabs, rounds = std::ceil(units / sm_count);
            const double time = rounds * (5000 + 11.0 * block_rows + 1.5 * d.nnz * pairs);
            if (time < least * 0.995) least = time, best = len;
        }
        return best;
    }
    int bwd_slot = -1, bwd_parts_done = 0, bwd_parts = 0;  // progress of a phased backward
    int fwd_slot = -1, fwd_parts_done = 0, fwd_parts = 0;  // progress of a forward pass run in pieces
    // peers of the fused data-parallel update: every rank's gradient and parameter buffer mapped here
    int xch_rank = -1, xch_world = 0;
    float* peer_g[b200::kMaxRanks] = {};
    float* peer_p[b200::kMaxRanks] = {};
    int* xch_flags = nullptr;  // this rank's fence counters (kernels_opt.cuh: PeerFlags)
    int* peer_flags[b200::kMaxRanks] = {};
    int xch_step = 0;          // fenced exchanges issued so far
    long long xch_spin_limit = b200::kPeerWaitSpins;
    int xch_wait_ready = 0;    // value the next exchange launch waits for at kFlagReady (0: the caller fences)
    bool xch_fenced_used = false;
    int* h_gave_up = nullptr;  // pinned: raised by a kernel whose wait for its own copies ran out
    int* h_xstatus = nullptr;  // pinned ring beside h_status: per update the fence time-out word and what was missing
    bool loss_in_param = false;  // the last update left the summed loss in P[0] instead of G[0]
    int exchange_ctas = 0;          // CTAs of a side-stream exchange launch (0: one per SM)
    // the exchange that runs under the feature-transformer backward (b200_step_exchange)
    cudaStream_t xch_stream = nullptr;  // highest priority: its few CTAs take their SMs before the backward's many
    cudaEvent_t xch_fork = nullptr, xch_join = nullptr;
    b200::PeerFlags* d_peers = nullptr;  // device copy of the peers' counter arrays, for the backward's CTAs
    int* done_count = nullptr;           // [nblocks] backward CTAs finished per row block
    float* facc = nullptr;               // running block sum of this rank's share of the factoriser gradient
    float* d_win_rate = nullptr;         // device-side preparation: sigmoid(score / scale) for every 16-bit score
    float win_rate_scale = 0.f;          // the scale the table was made for (0: none yet)
    float host_scale = 0.f;              // the scale of the records that came without a table, one after the other,
    int64_t host_positions = 0;          // and how many there were
    int* d_expanded = nullptr;           // [64] 768 * king bucket per square, and the layout it was made from
    int32_t expanded_layout[32] = {};
    bool expanded_valid = false;
    int overlap_ctas = 20;               // SMs the overlapped exchange occupies
    bool overlap_mode = false;           // batches are cut for a backward that runs beside the exchange
    bool sig_on = false;                 // the running backward announces finished row blocks
    int sig_value = 0;
    bool manual_grad_zero = false;  // the caller zeroes the gradient buffer range by range (b200_grad_zero_range)
    bool tiled_ok = false, tiled_promised = false;  // promised: what the caller may ask for by name (FT_TILED)
    bool have_backward = false;
    bool w1_dirty = true, merged_dirty = true;  // the weights moved since the regrouped first dense layer / the merged table was built
    bool trains = false;  // a training pass has run: uploads then also build what only the backward reads
    int nblocks = 1, nslabs = 1;
    int block_rows = 0;  // table rows per block: as promised, or a small table as a single block
    int last_n = 0;
    // per-step CUDA events on the compute stream, kept for the last kTimingRing steps
    static constexpr int kTimingRing = 256, kTimingEvents = 8;
    cudaEvent_t tev[kTimingRing][kTimingEvents] = {};
    int64_t steps_begun = 0, steps_done = 0, timing_origin = 0;
    bool events_made = false;
    // ... or, for whole steps (b200_step), time stamps that the kernels write themselves (launch.cuh)
    unsigned long long* d_stamps = nullptr;  // [kTimingRing][kTimingEvents]
    bool stamped[kTimingRing] = {};          // how the ring's entry was taken
    bool chained = false;                    // the launches being enqueued are one whole step's
    unsigned long long* stamp(int k) const { return chained ? d_stamps + (steps_begun % kTimingRing) * kTimingEvents + k : nullptr; }
    bool step_open = false;
    int64_t opt_step = 0;   // completed optimiser steps (RAdam's step count; reset when the rule changes)
    float* S = nullptr;     // Ranger's slow weights, same layout as P (allocated when a tensor first uses Ranger)
    int64_t launches = 0, h2d_bytes = 0;
    std::vector<void*> allocations;

    int* kept_bucket = nullptr;  // dense_one: the output bucket of every position of the last training pass
    int w1_now = 0;              // which of two copies of the regrouped weights is current; the last training pass may have used the other
    const float* w1_used = nullptr;  // the copy that the last training pass used
    int grad_n = 0;              // its positions (0: none has run)
    bool dx_formed = false;      // dx holds its gradient at x, which such a network forms only where somebody asks
    float* w1g_copy(int k) const { return w1g + (size_t)k * d.n_out_buckets * d.dense_out[0] * D1(); }
    int D1() const { return d.pairwise ? d.ft_out : 2 * d.ft_out; }
    int dense_in(int l) const { return l == 0 ? D1() : d.dense_out[l - 1]; }
    Tensor* find(const char* name) {
        for (auto& t : tensors)
            if (t.name == name) return &t;
        return nullptr;
    }
    // AUTO: both passes take the shared-memory kernels whenever the inputs allow it (measured
    // at 16384 positions, H = 2048: backward 0.50 ms against 0.61 ms for global vector reductions)
    bool fwd_tiled() const { return ft_fwd_mode == B200_FT_TILED || (ft_fwd_mode == B200_FT_AUTO && tiled_ok); }
    // ... for a whole batch of n positions.  The tiled forward stages every table row once whatever the batch holds, in few
    // CTAs when there are few pairs; the gather forward reads the rows of the batch only, from L2 (two per feature with a
    // factoriser).  Drawn for lists that are full, whose rows cost the gather twice as much and the tiled walk little more.
    // Forward kernel of a training step on a B200, us, gather / tiled, half of the slots active; all:
    //   with a factoriser, by rows of the batch over the table's: 768 x 16 rows, 2048 columns pairwise 2.1 57 / 79; 69 / 88, 2.9 62 / 76; 80 / 92, 3.4 66 / 78; 89 / 86
    //   1024 columns 2.1 25 / 41; 29 / 45, 2.9 33 / 37; 44 / 47, 3.4 34 / 37; 46 / 40; 128 columns 3.9 12 / 19; 13 / 21; 768 x 32 x 1024 3.0 55 / 69; 75 / 81, 3.9 62 / 75; 94 / 86
    //   768 x 10 x 1024 2.9 20 / 28; 26 / 30, 4.0 27 / 28; 40 / 32; 768 x 4 x 1024 4.0 16 / 18; 18 / 20, x 2048 pairwise 2.9 22 / 28; 25 / 30, 4.0 30 / 26; 37 / 29
    //   96 x 64 rows x 1024 3.9 19 / 35; 26 / 35, x 256 7 / 19; 8 / 19: the wider the table the sooner, as the tiles take a time of their own besides: below three times the
    //   rows by the more of a wide table, up to four times of a narrow one (the merged table begins at five)
    //   without, by MB of slots: 768 rows x 1024 columns 160 11.0 / 12.6; 12.5 / 15.0, 256 12.5 / 15.6; 16.5 / 17.8, 320 18.8 / 16.7; 26 / 20; 768 x 512 256 12.0 / 14.0; 15.3 / 17.5
    //   147 rows x 512 128 9.0 / 11.2; 11.4 / 13.2, 160 11 / 11.3; 13 / 12.2, 256 12.4 / 12.0; 14.7 / 14.6; x 2048 128 9.5 / 11.9; 11.5 / 13.6, 256 14.2 / 12.6; 16.3 / 14.7
    //   31 x 4 rows x 512 96 8.1 / 8.0; 9.7 / 10.1, 128 9.0 / 8.8; 11.3 / 10.2, 192 9.9 / 9.7; 12.0 / 12.1: the more rows a tile has the later
    bool fwd_tiled(int n) const {
        const long long rows = (long long)n * d.nnz;
        const int columns = d.ft_out > 512 ? (d.ft_out + 255) & ~255 : d.ft_out;  // as gather_shape's warps take them
        const bool gather = d.factoriser_rows ? rows < 4LL * d.n_inputs && (4 * rows - 11LL * d.n_inputs) * d.ft_out < kGatherMore
                                              : (long long)n * kGatherRowsPerPosition <= 4LL * d.n_inputs ||
                                                    (n <= 2048 && 8 * rows * columns <= kGatherMostBytes + kGatherMostPerRow * block_rows);
        return fwd_tiled() && !(ft_fwd_mode == B200_FT_AUTO && gather);
    }
    // The gather forward of n positions reads the merged table (one row per feature, after a pass over the whole table)
    // when the batch gathers several times the table's rows; below that it adds the factoriser row by row.
    bool merged_table(int n) const { return d.factoriser_rows && !fwd_tiled(n) && (long long)n * d.nnz >= 5LL * d.n_inputs; }
    float* w1g_now() const { return w1g ? w1g_copy(w1_now) : nullptr; }
    void weights_moved() { w1_dirty = merged_dirty = true; }
    bool bwd_tiled() const { return ft_bwd_mode == B200_FT_TILED || (ft_bwd_mode == B200_FT_AUTO && tiled_ok); }
    // the register-tiled dense forward (rows per bucket in fours, more layers after the first) also
    // forms the gradients of those later layers
    bool fused_small_grads() const { return dense_mma(); }
    // one row per bucket and nothing behind it (and rows that fit the kernel's stages): dense_one_kernel
    bool dense_one() const { return d.n_dense == 1 && D1() <= b200::kOneMaxK; }
    // such a network's x holds the roots of squared activations (activation 3 of kernels_ft.cuh)
    bool keep_root() const { return dense_one() && d.ft_act == B200_ACT_SCRELU; }
    // first dense layers of four and more rows per bucket run on the tensor pipe
    bool dense_mma() const { return d.dense_out[0] >= 4; }
    // Which batches of n positions ft_backward_mma_kernel takes: those it is the faster form for, of a table whose rows fit into one
    // tile, unless the backward has to announce finished row blocks or was asked for by another shape.
    bool small_table() const { return tiled_ok && block_rows < b200::kMmaTileRows; }
    bool bwd_mma(int n) const { return small_table() && bwd_wide && !overlap_mode && (bwd_products > 0 || (bwd_products < 0 && products_pay(n))); }
    // Both forms' ns for 128 pairs x 32 columns on one SM, fitted to the sweep below.  Products write out the whole tile whatever the
    // lists hold, cut every block's pairs into steps of its own (one more on average is not full) and take out its sums; the walk's time goes
    // with the active rows, of which the host knows the slots: half of them, as of the games' lists.  The line is drawn 1.4 times to the
    // walk's side, which also leaves it small batches, where a step's latency counts.  Backward on a B200, walk / products in us (rows x blocks, active of slots):
    //   147 x 1, 27 of 49: 32768 positions x 256 columns 83 / 41, 4096 x 1024 46 / 24, 512 x 64 11.0 / 9.6, 300 x 64 10.5 / 9.7 (walks), pairwise 16384 x 512 88 / 62
    //   255 x 1, 17 of 32: 32768 x 256 60 / 47, 4096 x 1024 34 / 28, 3000 x 128 9.7 / 12.5 (walks), pairwise 16384 x 512 66 / 75 (walks)
    //   255 x 1, 4 of 8: 32768 x 256 31 / 47 (walks);  64 x 1, 8 of 16: 32768 x 256 39 / 36.5, pairwise 16384 x 512 45 / 58 (walks)
    //   200 x 8, 17 of 32: 16384 x 256 32 / 28, 1024 x 2048 22 / 34 (walks), pairwise 32768 x 1024 235 / 252 (walks)
    //   147 x 64, 17 of 32: 16384 x 256 39.5 / 38 (given up), 1024 x 2048 41 / 131 (walks);  31 x 1000, 4 of 8: 1024 x 2048 293 / 762 (walks; with the walk of before)
    // Lists that are emptier than half may get the slower form: 255 rows, 4 of 32 slots, 32768 x 256 loses 13 of 98 us.
    bool products_pay(int n) const {
        const long long steps = ((long long)2 * n + b200::kStepPairs - 1) / b200::kStepPairs, blocks = std::min<long long>(nblocks, 2LL * n);
        const long long product = (d.pairwise ? 1700 : 900) + b200::ft_mma_rows(block_rows) * 22 / 10, walk = 900 + 85 * d.nnz / 2;
        return 14 * (steps + (1 + b200::kUnitFixed) * blocks) * product < 10 * steps * walk;
    }
    unsigned* gmax = nullptr;    // see FtArgs
    int fwd_last = 0;            // the last forward's kernel: 0 gather, 1 tiled, 2 tiled with the next tile fetched ahead
    bool products_last = false;  // the last backward was ft_backward_mma_kernel
    int chunk_last = 0;          // pairs per chunk of the last backward, 0: the gather
    bool update_copies = false;  // the last whole step's update took a warp per copy of the factoriser
};

namespace {

// The per-tensor table of the update kernels for the step that is being enqueued.  RAdam's step size and
// its "second moment divides yet" flag depend on the step count only and are evaluated here in fp32, as
// RAdam::update does on the host (radam.rs:295-314).
void fill_segments(const b200_net* net, b200::AdamArgs& a) {
    a.nseg = (int)net->tensors.size();
    for (int i = 0; i < a.nseg; i++) {
        const Tensor& t = net->tensors[i];
        b200::AdamSegment seg{t.off / 4, (t.off + t.n + 3) / 4, t.hp.decay, t.hp.beta1, t.hp.beta2, t.hp.min_weight, t.hp.max_weight};
        if (t.opt_kind != B200_OPT_ADAMW) {
            const float step = (float)(net->opt_step + 1);
            const float beta2_t = powf(t.hp.beta2, step);
            const float n_sma_max = 2.0f / (1.0f - t.hp.beta2) - 1.0f;
            const float n_sma = n_sma_max - 2.0f * step * beta2_t / (1.0f - beta2_t);
            const float denom = 1.0f - powf(t.hp.beta1, step);
            if (n_sma > t.n_sma_threshold) {
                const float p1 = (n_sma - 4.0f) / (n_sma_max - 4.0f), p2 = (n_sma - 2.0f) / n_sma, p3 = n_sma_max / (n_sma_max - 2.0f);
                seg.rate_scale = sqrtf((1.0f - beta2_t) * p1 * p2 * p3) / denom;
                seg.use_denom = 1;
            } else {
                seg.rate_scale = 1.0f / denom;
                seg.use_denom = 0;
            }
        }
        a.seg[i] = seg;
    }
}

int set_device(const b200_net* net) {
    CK(cudaSetDevice(net->device));
    return 0;
}

template <class T>
int dev_alloc(b200_net* net, T** p, size_t count) {
    void* raw = nullptr;
    if (cudaMalloc(&raw, std::max<size_t>(count, 1) * sizeof(T)) != cudaSuccess) {  // once more without what the operator's pool keeps
        cudaGetLastError();
        b200::op_pool_trim(net->device);
        CK(cudaMalloc(&raw, std::max<size_t>(count, 1) * sizeof(T)));
    }
    net->allocations.push_back(raw);
    *p = static_cast<T*>(raw);
    return 0;
}

// Device buffers to be taken from one allocation.
struct Plan {
    struct Item {
        void** p;
        size_t bytes;
    };
    std::vector<Item> items;
    template <class T>
    void add(T** p, size_t count) {
        items.push_back({reinterpret_cast<void**>(p), align_up(std::max<size_t>(count, 1) * sizeof(T), 256)});
    }
    int allocate(b200_net* net) {
        size_t total = 0;
        for (const Item& i : items) total += i.bytes;
        char* base = nullptr;
        if (int rc = dev_alloc(net, &base, total)) return rc;
        for (const Item& i : items) {
            *i.p = base;
            base += i.bytes;
        }
        return 0;
    }
};

bool supported_m(int m) { return m == 1 || m == 2 || m == 4 || m == 8 || m == 16 || m == 32; }

int validate(const b200_net_desc& d) {
    if (d.n_inputs < 1 || d.n_inputs > 65534) return b200::fail(B200_ERR_UNSUPPORTED, "n_inputs must be in [1, 65534]");
    if (d.nnz < 1 || d.nnz > 64) return b200::fail(B200_ERR_UNSUPPORTED, "nnz must be in [1, 64]");
    if (d.ft_out < 8 || d.ft_out % 8) return b200::fail(B200_ERR_UNSUPPORTED, "ft_out must be a positive multiple of 8");
    if (d.ft_act != B200_ACT_CRELU && d.ft_act != B200_ACT_SCRELU)
        return b200::fail(B200_ERR_UNSUPPORTED, "ft_act must be CReLU or SCReLU");
    if (d.pairwise && d.ft_act != B200_ACT_CRELU) return b200::fail(B200_ERR_UNSUPPORTED, "pairwise_mul needs CReLU");
    if (d.factoriser_rows < 0 || (d.factoriser_rows && d.n_inputs % d.factoriser_rows))
        return b200::fail(B200_ERR_ARG, "factoriser_rows must tile n_inputs");
    if (d.n_out_buckets < 1 || d.n_out_buckets > 64) return b200::fail(B200_ERR_UNSUPPORTED, "1..64 output buckets");
    if (d.n_dense < 1 || d.n_dense > 3) return b200::fail(B200_ERR_UNSUPPORTED, "one to three dense layers");
    for (int l = 0; l < d.n_dense; l++) {
        if (d.dense_out[l] < 1 || d.dense_out[l] > 32 || (l == 0 && !supported_m(d.dense_out[l])))
            return b200::fail(B200_ERR_UNSUPPORTED, "dense layer %d: rows per bucket must be 1,2,4,8,16 or 32", l + 1);
        if (d.dense_act[l] < 0 || d.dense_act[l] > 2) return b200::fail(B200_ERR_ARG, "dense layer %d: bad activation", l + 1);
    }
    for (int l = 1; l < d.n_dense; l++)
        if (!supported_m(d.dense_out[l])) return b200::fail(B200_ERR_UNSUPPORTED, "dense layer %d: rows per bucket must be a power of two <= 32", l + 1);
    if (d.dense_out[d.n_dense - 1] != 1 || d.dense_act[d.n_dense - 1] != B200_ACT_NONE)
        return b200::fail(B200_ERR_UNSUPPORTED, "the last dense layer must have one row per bucket and no activation");
    if (d.max_batch < 1) return b200::fail(B200_ERR_ARG, "max_batch must be positive");
    if (d.ft_block_rows < 0) return b200::fail(B200_ERR_ARG, "ft_block_rows must not be negative");
    return 0;
}

void slot_layout(const b200_net* net, Slot& s, int n) {
    const b200_net_desc& d = net->d;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t at = off;
        off = align_up(off + bytes, 256);
        return at;
    };
    const size_t nb = net->nblocks, O = d.n_out_buckets, bins = nb + O;
    const bool many = net->nblocks > b200::kGroupMaxBlocks;
    s.off_stm = take((size_t)n * d.nnz * 2);
    s.off_nstm = take((size_t)n * d.nnz * 2);
    s.off_buckets = take((size_t)n * 4);
    s.off_targets = take((size_t)n * 4);
    s.off_order = take((size_t)n * 4);
    s.off_dtiles = take(((size_t)n / b200::kDenseTile + O + 1) * 8);
    s.off_records = take((size_t)n * 36);  // and, of some batches, their targets
    s.off_pairs = take((size_t)n * 16);
    s.off_blocks = take((nb + 1) * 4);
    s.off_chunks = take(((size_t)2 * n / b200::kChunkLeast + nb + 1) * 16);
    s.off_cbegin = take((nb + 1) * 4);
    s.off_bexpect = take(nb * 4);
    s.off_status = take(4);
    s.off_info = take((size_t)n * 8);
    s.off_hist = take(many ? 4 : (size_t)(b200::group_ctas(n) + 1) * bins * 4);
    s.off_many[0] = take(many ? bins * 4 : 4);
    s.off_many[1] = take(many ? (bins + 2) * 4 : 4);
    s.off_many[2] = take(many ? (bins + 1) * 4 : 4);
    s.bytes = off;
}

template <bool PW>
int launch_ft_forward(b200_net* net, const b200::FtArgs& a, const b200::TileArgs& t, bool tiled, int grid) {
    const bool ahead = tiled && b200::ft_fwd_ahead(a, t, grid);
    net->fwd_last = tiled ? ahead ? 2 : 1 : 0;
    if (tiled) {
        CK(b200::launch_step(false, ahead ? b200::ft_forward_tiled_kernel<PW, true> : b200::ft_forward_tiled_kernel<PW, false>, grid, b200::kFwdThreads, b200::ft_fwd_smem(t.block_rows, t.list_len), net->stream, a, t));
    } else {
        const b200::GatherShape g = b200::gather_shape(a.n, PW ? a.H / 2 : a.H, PW, a.factor != nullptr, net->sm_count);
        (a.factor ? b200::gather_form<PW, true>(g) : b200::gather_form<PW, false>(g))<<<g.grid, 256, 0, net->stream>>>(a, g.pairs);
    }
    LAUNCHED(net);
    return 0;
}

template <bool PW, bool ONE>
void launch_ft_backward_tiled(const b200::FtArgs& a, const b200::TileArgs& t, bool wide, int grid, size_t smem, bool chained, cudaStream_t stream) {
    // data-parallel runs that announce finished row blocks take an instantiation of their own: the
    // fence it ends with makes every CTA wait for its reductions to land (measured: +18 %)
    if (wide && t.sig.done_count)
        b200::launch_step(chained, b200::ft_backward_tiled_kernel<PW, 1024, true, ONE>, grid, 1024, smem, stream, a, t);
    else if (wide)
        b200::launch_step(chained, b200::ft_backward_tiled_kernel<PW, 1024, false, ONE>, grid, 1024, smem, stream, a, t);
    else if (t.sig.done_count)
        b200::launch_step(chained, b200::ft_backward_tiled_kernel<PW, 512, true, ONE>, grid, 512, smem, stream, a, t);
    else
        b200::launch_step(chained, b200::ft_backward_tiled_kernel<PW, 512, false, ONE>, grid, 512, smem, stream, a, t);
}

// the one of its forms that a network takes
void (*ft_backward_mma(const b200_net* net))(b200::FtArgs, b200::TileArgs) {
    const bool one = net->dense_one();
    if (net->d.pairwise) return one ? b200::ft_backward_mma_kernel<true, true, false> : b200::ft_backward_mma_kernel<true, false, false>;
    if (net->d.ft_act == B200_ACT_CRELU) return one ? b200::ft_backward_mma_kernel<false, true, false> : b200::ft_backward_mma_kernel<false, false, false>;
    return one ? b200::ft_backward_mma_kernel<false, true, true> : b200::ft_backward_mma_kernel<false, false, true>;
}

template <bool PW>
int launch_ft_backward(b200_net* net, const Slot& s, const b200::FtArgs& a, const b200::TileArgs& t, bool tiled, int grid) {
    net->products_last = tiled && s.mma;
    net->chunk_last = tiled ? t.chunk_len : 0;
    if (tiled && s.mma) {
        b200::launch_step(net->chained, ft_backward_mma(net), grid, b200::kMmaThreads, b200::ft_mma_smem(b200::ft_mma_rows(t.block_rows)), net->stream, a, t);
    } else if (tiled) {
        const size_t smem = b200::ft_bwd_smem(t.block_rows, a.nnz, t.chunk_len);
        const bool wide = t.wide;
        if (net->dense_one()) launch_ft_backward_tiled<PW, true>(a, t, wide, grid, smem, net->chained, net->stream);
        else launch_ft_backward_tiled<PW, false>(a, t, wide, grid, smem, net->chained, net->stream);
    } else {
        const int unit = PW ? a.H / 2 : a.H;
        dim3 grid((2 * a.n + 63) / 64, (unit + 127) / 128);
        if (net->dense_one()) b200::launch_step(net->chained, b200::ft_backward_gather_kernel<PW, true>, grid, 256, 0, net->stream, a, 64);
        else b200::launch_step(net->chained, b200::ft_backward_gather_kernel<PW, false>, grid, 256, 0, net->stream, a, 64);
    }
    LAUNCHED(net);
    return 0;
}

// the layers of fewer than four rows, which the fp32 kernels take
#define DISPATCH_M12(m, ...)                                                  \
    switch (m) {                                                              \
        case 1: { constexpr int MM = 1; __VA_ARGS__; } break;                 \
        case 2: { constexpr int MM = 2; __VA_ARGS__; } break;                 \
        default: return b200::fail(B200_ERR_UNSUPPORTED, "rows per bucket %d", m); \
    }
#define DISPATCH_M(m, ...)                                                    \
    switch (m) {                                                              \
        case 1: { constexpr int MM = 1; __VA_ARGS__; } break;                 \
        case 2: { constexpr int MM = 2; __VA_ARGS__; } break;                 \
        case 4: { constexpr int MM = 4; __VA_ARGS__; } break;                 \
        case 8: { constexpr int MM = 8; __VA_ARGS__; } break;                 \
        case 16: { constexpr int MM = 16; __VA_ARGS__; } break;               \
        case 32: { constexpr int MM = 32; __VA_ARGS__; } break;               \
        default: return b200::fail(B200_ERR_UNSUPPORTED, "rows per bucket %d", m); \
    }

// A slice of a tile is a chain of sixteen rounds of loads for its warp: while there are fewer of them than warps, up to eight
// warps share one (but none is left without a group of columns).
int dense_slices(const b200_net* net) { return (net->D1() + b200::kSliceCols - 1) / b200::kSliceCols; }
int dense_split(const b200_net* net, int ntiles) {
    const int slices = dense_slices(net), all = b200::kSliceCols / b200::kMmaCols;
    const int in_last = (net->D1() + b200::kMmaCols - 1) / b200::kMmaCols - (slices - 1) * all;
    int split = 8;
    while (split > 1 && ((long long)slices * split * ntiles > 8LL * net->sm_count || (split - 1) * (all / split) >= in_last)) split /= 2;
    return split;
}

template <int MM>
void launch_dense_forward(b200_net* net, const b200::DenseArgs& da, int ntiles) {
    if constexpr (MM >= 4) {
        const int slices = dense_slices(net), split = dense_split(net, ntiles);
        const dim3 grid(slices, std::max(1, std::min((ntiles * split + 7) / 8, b200::dense_mma_ctas(MM) * net->sm_count / slices)));
        b200::launch_step(net->chained, b200::dense_first_mma_kernel<MM>, grid, 256, b200::dense_mma_smem<MM>(), net->stream, da, split);
        net->launches++;
        b200::launch_step(net->chained, b200::dense_small_mma_kernel<MM>, std::min(ntiles, b200::kSmallCtas * net->sm_count), b200::kSmallThreads, 0, net->stream, da,
                          slices * split);
    } else
        b200::launch_step(net->chained, b200::dense_forward_kernel<MM>, ntiles, 256, b200::dense_fwd_smem<MM>(), net->stream, da);
}
template <int MM>
void launch_wgrad_mma(b200_net* net, const b200::DenseArgs& a, float* gW) {
    if constexpr (MM >= 4) {
        const int cols = 8 * b200::kWgradCols, gx = (a.K1 + cols - 1) / cols;
        const dim3 grid(gx, std::max(1, std::min(a.ntiles, b200::dense_mma_ctas(MM) * net->sm_count / gx)));
        b200::launch_step(net->chained, b200::dense_wgrad_mma_kernel<MM>, grid, b200::kRingThreads, b200::wgrad_smem<MM>(), net->stream, a, gW);
    }
}
template <int MM>
void launch_dense_dx(b200_net* net, const b200::DenseArgs& da, int ntiles) {
    if constexpr (MM >= 4)
        b200::launch_step(net->chained, b200::dense_dx_mma_kernel<MM>, ntiles, 256, 0, net->stream, da, net->dx);
    else
        b200::launch_step(net->chained, b200::dense_dx_kernel<MM>, ntiles, 256, 0, net->stream, da, net->dx);
}

template <int MM>
cudaError_t set_dense_forward_smem() {
    if constexpr (MM >= 4)
    {
        const cudaError_t e = b200::allow_smem(b200::dense_first_mma_kernel<MM>);
        return e ? e : b200::allow_smem(b200::dense_wgrad_mma_kernel<MM>);
    } else
        return b200::allow_smem(b200::dense_forward_kernel<MM>);
}

// Most chunks that a batch of n positions can be cut into: every block may end in a partly filled one.
int most_chunks(const b200_net* net, int n, int chunk_len) { return std::min(2 * n, 2 * n / chunk_len + net->nblocks); }

// Grid of the tiled kernels: one CTA per SM (two for the 512-thread backward), fewer when there is too little work to give
// every CTA a worthwhile piece.  What a run of row blocks holds is known on the device only: a CTA without work returns.
int ft_forward_grid(const b200_net* net, const Slot& s) {
    const long long line = (long long)net->nslabs * 2 * s.n;
    return (int)std::max<long long>(1, std::min<long long>(net->sm_count, line / kMinItemPairs));
}
int ft_backward_grid(const b200_net* net, const Slot& s, bool beside_exchange) {
    const long long units = (long long)net->nslabs * s.n_chunks * (s.mma ? 2 : 1);
    const int per_sm = s.wide ? 1 : 2;
    const int sms = net->sm_count - (beside_exchange ? std::min(net->overlap_ctas, net->sm_count - 1) : 0);
    return (int)std::max<long long>(1, std::min<long long>((long long)sms * per_sm, units));
}

b200::FtArgs ft_args(b200_net* net, const Slot& s) {
    b200::FtArgs a{};
    const b200_net_desc& d = net->d;
    // the tiled forward adds the factoriser while it fills its tile; only the gather forward of a large batch
    // needs the merged table
    const bool merged = net->merged_table(s.n);
    a.table = merged ? net->table : net->P + net->find("l0w")->off;
    a.factor = (net->d.factoriser_rows && !merged) ? net->P + net->find("l0f")->off : nullptr;
    a.factor_rows = net->d.factoriser_rows;
    a.block_rows = net->ft_fwd_mode == B200_FT_AUTO && net->tiled_ok ? net->block_rows : 0;
    a.bias = net->P + net->find("l0b")->off;
    a.idx_stm = s.dev<uint16_t>(s.off_stm);
    a.idx_nstm = s.dev<uint16_t>(s.off_nstm);
    a.n = s.n;
    a.nnz = d.nnz;
    a.H = d.ft_out;
    a.n_inputs = d.n_inputs;
    a.act = net->keep_root() ? 3 : d.ft_act;
    a.x = net->x;
    a.u = net->u;
    a.dx = net->dx;
    a.w1 = net->w1_used;
    a.dout = net->dz[0];
    a.out_bucket = net->kept_bucket;
    a.stamp = nullptr;
    a.gmax = s.mma ? net->gmax : nullptr;
    a.gave_up = net->h_gave_up;
    a.g_table = net->G + net->find("l0w")->off;
    a.g_bias = net->G + net->find("l0b")->off;
    return a;
}

b200::TileArgs tile_args(b200_net* net, const Slot& s, bool backward) {
    b200::TileArgs t{};
    t.block_rows = net->block_rows;
    t.nslabs = net->nslabs;
    t.first_block = 0;
    t.last_block = net->nblocks;
    t.chunk_begin = s.dev<int>(s.off_cbegin);
    t.pairs = s.dev<int2>(s.off_pairs);
    t.block_begin = s.dev<int>(s.off_blocks);
    t.status = s.dev<int>(s.off_status);
    t.lists = s.lists;
    t.list_len = (net->d.nnz + 7) & ~7;
    t.walk_warps = b200::ft_fwd_warps(net->block_rows, t.list_len);
    t.fill_steps = (t.block_rows + b200::kFwdThreads / 8 - 1) / (b200::kFwdThreads / 8);
    t.chunks = s.dev<int4>(s.off_chunks);
    t.csr_ent = s.csr_ent;
    t.csr_start = s.csr_start;
    t.chunk_len = s.chunk_len;
    t.wide = s.wide;
    t.ent_cap = s.mma ? b200::ft_mma_ent_cap(net->block_rows) : b200::ft_bwd_ent_cap(net->block_rows, net->d.nnz, s.chunk_len);
    t.start_cap = s.mma ? b200::kStepHead : b200::ft_bwd_start_cap(net->block_rows, net->d.nnz, s.chunk_len);
    if (backward && net->sig_on) {
        t.sig.done_count = net->done_count;
        t.sig.done_expect = s.dev<int>(s.off_bexpect);
        t.sig.peers = net->d_peers;
        t.sig.value = net->sig_value;
    }
    return t;
}

b200::DenseArgs dense_args(b200_net* net, const Slot& s, bool want_grad) {
    b200::DenseArgs a{};
    const b200_net_desc& d = net->d;
    a.x = net->x;
    a.buckets = s.dev<int>(s.off_buckets);
    a.targets = s.dev<float>(s.off_targets);
    a.n = s.n;
    a.K1 = net->D1();
    a.O = d.n_out_buckets;
    a.n_dense = d.n_dense;
    for (int l = 0; l < d.n_dense; l++) {
        a.M[l] = d.dense_out[l];
        a.act[l] = d.dense_act[l];
        char name[16];
        snprintf(name, sizeof name, "l%dw", l + 1);
        a.W[l] = net->P + net->find(name)->off;
        snprintf(name, sizeof name, "l%db", l + 1);
        a.B[l] = net->P + net->find(name)->off;
        a.dz[l] = net->dz[l];
    }
    a.order = d.n_out_buckets > 1 ? s.dev<int>(s.off_order) : nullptr;
    a.tiles = d.n_out_buckets > 1 ? s.dev<int2>(s.off_dtiles) : nullptr;
    a.ntiles = s.n_dtiles;
    a.W1g = net->w1g_now();
    a.W1f = net->w1f;
    a.W1d = net->w1d;
    a.partial = net->dense_partial;
    a.dz_frag = net->dz_frag;
    a.gave_up = net->h_gave_up;
    a.gmax = want_grad && s.mma ? net->gmax : nullptr;  // (the walk needs no scale: up to 4 us of the dense kernels)
    a.a1 = net->a1;
    a.a2 = net->a2;
    a.out = net->out;
    a.out_host = !want_grad && s.n <= kDirectOutputs ? net->h_out : nullptr;
    a.loss = net->G;
    a.want_grad = want_grad ? 1 : 0;
    for (int l = 0; l < d.n_dense; l++) {
        char name[16];
        snprintf(name, sizeof name, "l%dw", l + 1);
        a.gW[l] = net->G + net->find(name)->off;
        snprintf(name, sizeof name, "l%db", l + 1);
        a.gB[l] = net->G + net->find(name)->off;
    }
    return a;
}

// dense_one: the gradient at x of the last training pass, for inspection (the backward forms it where it uses it)
int form_dx(b200_net* net) {
    if (net->grad_n < 1 || net->dx_formed) return 0;
    b200::dense_one_dx_kernel<<<net->sm_count * 8, 256, 0, net->stream>>>(net->w1_used, net->dz[0], net->kept_bucket, net->dx, net->grad_n, net->D1());
    LAUNCHED(net);
    net->dx_formed = true;
    return 0;
}

int refresh_table(b200_net* net, int n) {
    if (net->merged_dirty && net->merged_table(n)) {
        const Tensor* w = net->find("l0w");
        const Tensor* f = net->find("l0f");
        const size_t n4 = (size_t)w->n / 4, block4 = (size_t)f->n / 4;
        b200::factoriser_merge_kernel<<<net->sm_count * 8, 256, 0, net->stream>>>(
            reinterpret_cast<const float4*>(net->P + w->off), reinterpret_cast<const float4*>(net->P + f->off),
            reinterpret_cast<float4*>(net->table), n4, block4);
        LAUNCHED(net);
        net->merged_dirty = false;
    }
    if (net->w1_dirty) {
        const Tensor* w1 = net->find("l1w");
        const int O = net->d.n_out_buckets, M1 = net->d.dense_out[0];
        if (net->dense_mma()) {
            const int quads = (int)(b200::mma_table_words(net->D1(), O, M1) / 6);  // (a thread writes six words of each table)
            b200::dense_fragments_kernel<<<std::min(net->sm_count * 4, (quads + 255) / 256), 256, 0, net->stream>>>(
                net->P + w1->off, net->w1f, net->w1d, net->D1(), O, M1);
        } else {
            net->w1_now ^= 1;
            if (net->w1g_now() == net->w1_used)  // (only if the weights moved twice since the last training pass)
                if (int rc = form_dx(net)) return rc;
            b200::dense_regroup_kernel<<<std::min<int>(net->sm_count * 4, (int)((w1->n + 255) / 256)), 256, 0, net->stream>>>(
                net->P + w1->off, net->w1g_now(), net->D1(), O, M1);
        }
        LAUNCHED(net);
        net->w1_dirty = false;
    }
    return 0;
}

int check_slot(b200_net* net, int slot, const char* who) {
    if (!net) return b200::fail(B200_ERR_ARG, "%s: null net", who);
    if (slot < 0 || slot >= B200_NUM_SLOTS) return b200::fail(B200_ERR_ARG, "%s: slot %d out of range", who, slot);
    if (net->slots[slot].n < 1 || !net->slots[slot].has_ready)
        return b200::fail(B200_ERR_STATE, "%s: slot %d holds no batch", who, slot);
    return 0;
}

b200::GroupArgs group_args(b200_net* net, Slot& s, bool want_lists, bool want_order) {
    const b200_net_desc& d = net->d;
    b200::GroupArgs g{};
    g.stm = s.dev<uint16_t>(s.off_stm);
    g.nstm = s.dev<uint16_t>(s.off_nstm);
    g.buckets = s.dev<int>(s.off_buckets);
    g.n = s.n;
    g.nnz = d.nnz;
    g.n_inputs = d.n_inputs;
    g.block_rows = net->tiled_ok ? net->block_rows : d.n_inputs;
    g.nblocks = net->nblocks;
    g.n_out_buckets = d.n_out_buckets;
    g.info = s.dev<int>(s.off_info);
    g.hist = s.dev<int>(s.off_hist);
    g.status = s.dev<int>(s.off_status);
    g.clear_status = 1;
    g.want_lists = want_lists;
    g.nslabs = net->nslabs;
    if (want_lists) {
        g.pairs = s.dev<int2>(s.off_pairs);
        g.lists = s.lists;
        g.list_len = (d.nnz + 7) & ~7;
        g.block_begin = s.dev<int>(s.off_blocks);
        g.chunks = s.dev<int4>(s.off_chunks);
        g.chunk_begin = s.dev<int>(s.off_cbegin);
        g.max_chunks = s.n_chunks;
        g.chunk_len = s.chunk_len;
        g.expect = s.dev<int>(s.off_bexpect);
        g.expect_grid = s.expect_grid;
    }
    if (want_order) {
        g.order = s.dev<int>(s.off_order);
        g.tiles = s.dev<int2>(s.off_dtiles);
        g.max_tiles = s.n_dtiles;
    }
    return g;
}

// How the slot's batch is cut; the device fills the tables in.  The dense kernels' tiles at upload, what the tiled kernels
// take whenever their lists are built.
void cut_dense(b200_net* net, Slot& s) {
    const int O = net->d.n_out_buckets;
    s.n_dtiles = O > 1 ? s.n / b200::kDenseTile + std::min(O, s.n) : (s.n + b200::kDenseTile - 1) / b200::kDenseTile;
}
void cut_ft(b200_net* net, Slot& s) {
    if (!net->tiled_ok) return;
    s.wide = net->bwd_wide;
    s.mma = net->bwd_mma(s.n);
    s.chunk_len = s.mma ? b200::kStepPairs : net->bwd_chunk(s.n);
    s.n_chunks = most_chunks(net, s.n, s.chunk_len);
    s.expect_grid = s.mma ? 0 : ft_backward_grid(net, s, net->overlap_mode);
}

// Groups the slot's batch on `stream` (kernels_group.cuh); `counted`: the first pass has run with the featuriser.
int group_slot(b200_net* net, Slot& s, const b200::GroupArgs& g, bool counted, cudaStream_t stream) {
    if (g.nblocks > b200::kGroupMaxBlocks) {
        int *count = s.dev<int>(s.off_many[0]), *at = s.dev<int>(s.off_many[1]), *scratch = s.dev<int>(s.off_many[2]);
        const int pairs = (2 * g.n + 7) / 8;
        CK(cudaMemsetAsync(count, 0, (size_t)(g.nblocks + g.n_out_buckets) * sizeof(int), stream));
        b200::group_many_count_kernel<<<pairs, 256, 0, stream>>>(g, count);
        LAUNCHED(net);
        b200::group_many_scan_kernel<<<1, 1024, 0, stream>>>(g, count, at, scratch);
        LAUNCHED(net);
        b200::group_many_place_kernel<<<pairs, 256, 0, stream>>>(g, count);
        LAUNCHED(net);
    } else {
        const bool vec = b200::group_vec(g);
        // beside a training step a kernel that waits for the one before would hold its SMs meanwhile
        const bool chained = !net->trains;
        if (!counted) {
            b200::group_lists_kernel<<<b200::group_ctas(g.n), b200::kGroupThreads, 0, stream>>>(g, vec);
            LAUNCHED(net);
        }
        const bool scans = b200::group_scans(g.n);
        if (scans) {
            const int bins = g.nblocks + g.n_out_buckets;
            CK(b200::launch_step(chained, b200::group_scan_kernel, bins, 1024, 0, stream, g.hist, b200::group_ctas(g.n), bins));
            LAUNCHED(net);
        }
        CK(b200::launch_step(chained, b200::group_place_kernel, b200::group_windows(g.n), b200::kPlaceThreads, 0, stream, g, (int)vec, (int)scans));
        LAUNCHED(net);
    }
    if (g.want_lists) s.prepared = true;
    return 0;
}

int build_csr(b200_net* net, Slot& s, cudaStream_t stream) {
    if (s.mma)
        b200::ft_onehot_kernel<<<s.n_chunks, b200::kOnehotThreads, 0, stream>>>(tile_args(net, s, true));
    else
        b200::ft_csr_kernel<<<s.n_chunks, b200::kCsrThreads, b200::ft_csr_smem(net->block_rows, net->d.nnz, s.chunk_len), stream>>>(
            ft_args(net, s), tile_args(net, s, true));
    LAUNCHED(net);
    s.csr_built = true;
    return 0;
}

// The forward pass in three pieces: the per-pair row lists, the feature-transformer items of a
// run of work items, and the dense layers.
int forward_prepare(b200_net* net, Slot& s, bool want_grad) {
    // (a training pass wants the lists whenever its kernels may be the tiled ones, also where a small batch then takes the
    // gather forward: they report features outside their block, and the forward may be run in parts, which are tiled)
    const bool needed = want_grad ? net->fwd_tiled() || net->bwd_tiled() : net->fwd_tiled(s.n);
    if (needed && !s.prepared) {  // normally built at upload; here on the first training pass or after a change of kernels
        cut_ft(net, s);
        if (int rc = group_slot(net, s, group_args(net, s, true, false), false, net->stream)) return rc;
    }
    if (want_grad) net->status_slot = needed ? (int)(&s - net->slots) : -1;
    if (want_grad && !net->chained) CK(cudaEventRecord(net->tev[net->steps_begun % b200_net::kTimingRing][0], net->stream));
    return 0;
}

int forward_ft_blocks(b200_net* net, Slot& s, int first_block, int last_block) {
    const bool whole = first_block == 0 && last_block == net->nblocks;
    const bool tiled = whole ? net->fwd_tiled(s.n) : net->fwd_tiled();
    b200::FtArgs fa = ft_args(net, s);
    b200::TileArgs ta = tile_args(net, s, false);
    int grid = 0;
    if (tiled) {
        ta.first_block = first_block;
        ta.last_block = last_block;
        grid = ft_forward_grid(net, s);
    }
    return net->d.pairwise ? launch_ft_forward<true>(net, fa, ta, tiled, grid) : launch_ft_forward<false>(net, fa, ta, tiled, grid);
}

void (*dense_one_form(const b200_net* net, bool scale))(b200::OneArgs) {
    if (net->keep_root()) return scale ? b200::dense_one_kernel<true, true> : b200::dense_one_kernel<true, false>;
    return scale ? b200::dense_one_kernel<false, true> : b200::dense_one_kernel<false, false>;
}

int forward_dense(b200_net* net, Slot& s, bool want_grad) {
    if (want_grad && !net->chained) CK(cudaEventRecord(net->tev[net->steps_begun % b200_net::kTimingRing][1], net->stream));
    if (net->zero_pending) {  // the loss and every gradient from here on land in the cleared buffer
        CK(cudaStreamWaitEvent(net->stream, net->zero_done, 0));
        net->zero_pending = false;
    }
    b200::DenseArgs da = dense_args(net, s, want_grad);
    da.stamp = net->stamp(1);
    if (net->dense_one()) {
        b200::OneArgs a{};
        a.x = da.x, a.buckets = da.buckets, a.targets = da.targets, a.order = da.order, a.tiles = da.tiles;
        a.n = da.n, a.ntiles = da.ntiles, a.K1 = da.K1, a.O = da.O;
        a.W = da.W1g, a.B = da.B[0];
        a.dout = net->dz[0], a.kept_bucket = net->kept_bucket, a.out = da.out, a.out_host = da.out_host, a.loss = da.loss;
        a.gW = net->G + net->find("l1w")->off, a.gB = net->G + net->find("l1b")->off;
        a.want_grad = da.want_grad;
        a.stamp = da.stamp;
        a.gave_up = net->h_gave_up;
        a.gmax = da.gmax;
        if (want_grad) net->w1_used = da.W1g, net->grad_n = s.n, net->dx_formed = false;
        const size_t smem = b200::one_smem(a.K1);
        const int units = a.ntiles * (b200::kDenseTile / b200::one_rows(a.K1)), slots = net->sm_count * std::max(1, std::min(4, (int)(220 * 1024 / smem)));
        a.units_per_run = (units + slots - 1) / slots;
        b200::launch_step(net->chained, dense_one_form(net, a.gmax != nullptr), (units + a.units_per_run - 1) / a.units_per_run, b200::kOneThreads, smem, net->stream, a);
        LAUNCHED(net);
        return 0;
    }
    DISPATCH_M(net->d.dense_out[0], launch_dense_forward<MM>(net, da, s.n_dtiles));
    LAUNCHED(net);
    return 0;
}

int forward_part(b200_net* net, Slot& s, bool want_grad) {
    if (int rc = forward_prepare(net, s, want_grad)) return rc;
    if (int rc = forward_ft_blocks(net, s, 0, net->nblocks)) return rc;
    return forward_dense(net, s, want_grad);
}

int launch_wgrad(b200_net* net, const Slot& s) {
    const b200_net_desc& d = net->d;
    float *gW = net->G + net->find("l1w")->off, *gB = net->G + net->find("l1b")->off;
    if (net->dense_mma()) {
        const b200::DenseArgs a = dense_args(net, s, true);
        DISPATCH_M(d.dense_out[0], launch_wgrad_mma<MM>(net, a, gW));
        LAUNCHED(net);
        return 0;
    }
    b200::WgradArgs w{};
    w.X = net->x;
    w.dY = net->dz[0];
    w.order = d.n_out_buckets > 1 ? s.dev<int>(s.off_order) : nullptr;
    w.buckets = s.dev<int>(s.off_buckets);
    w.n = s.n;
    w.K = net->dense_in(0);
    w.O = d.n_out_buckets;
    w.gW = gW;
    w.gB = gB;
    const int groups = w.K / 4 + 1;  // four columns per thread, plus the bias
    const int threads = groups >= 128 ? 128 : ((groups + 31) / 32) * 32;
    const int gx = (groups + threads - 1) / threads;
    // The grid should fill the CTA slots the device offers exactly once or twice: a few CTAs
    // left over for another wave would double the kernel's time.
    if (!net->wgrad_per_sm) {
        int per_sm = 0;
        DISPATCH_M12(d.dense_out[0], cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, b200::dense_wgrad_kernel<MM>, threads, 0));
        net->wgrad_per_sm = std::max(1, per_sm);
    }
    const int slots = net->wgrad_per_sm * net->sm_count;
    const int waves = s.n >= 65536 ? 2 : 1;
    int chunks = std::max(1, std::min((s.n + 31) / 32, waves * slots / gx));
    w.chunk_len = (s.n + chunks - 1) / chunks;
    chunks = (s.n + w.chunk_len - 1) / w.chunk_len;
    dim3 grid(gx, chunks);
    DISPATCH_M12(d.dense_out[0], b200::launch_step(net->chained, b200::dense_wgrad_kernel<MM>, grid, threads, 0, net->stream, w));
    LAUNCHED(net);
    return 0;
}

// Weight and bias gradients of every dense layer.  They need the forward pass and the loss
// gradient only, so they run before the feature-transformer backward: once that ends, every
// gradient outside l0w is complete as well.
int launch_dense_grads(b200_net* net, Slot& s) {
    const b200_net_desc& d = net->d;
    if (net->d.n_dense > 1 && !net->fused_small_grads()) {  // the narrow layers' weight and bias gradients, one launch
        b200::SmallGradArgs g{};
        g.order = d.n_out_buckets > 1 ? s.dev<int>(s.off_order) : nullptr;
        g.tiles = d.n_out_buckets > 1 ? s.dev<int2>(s.off_dtiles) : nullptr;
        g.buckets = s.dev<int>(s.off_buckets);
        g.n = s.n;
        g.O = d.n_out_buckets;
        g.n_layers = d.n_dense - 1;
        for (int l = 1; l < d.n_dense; l++) {
            char name[16];
            g.K[l - 1] = d.dense_out[l - 1];
            g.M[l - 1] = d.dense_out[l];
            g.X[l - 1] = l == 1 ? net->a1 : net->a2;
            g.dY[l - 1] = net->dz[l];
            snprintf(name, sizeof name, "l%dw", l + 1);
            g.gW[l - 1] = net->G + net->find(name)->off;
            snprintf(name, sizeof name, "l%db", l + 1);
            g.gB[l - 1] = net->G + net->find(name)->off;
        }
        b200::launch_step(net->chained, b200::dense_small_grads_kernel, s.n_dtiles, 256, 0, net->stream, g);
        LAUNCHED(net);
    }
    return launch_wgrad(net, s);
}

// With lazy module loading (the CUDA default) a kernel's code reaches the GPU at its first launch, and
// that load can wait for running kernels to finish.  The data-parallel exchange has kernels that wait,
// bounded, for other kernels launched after them, so no kernel of this library may be loaded for the
// first time while one of those is spinning: load them all when the network is created.
template <class K>
bool load_kernel(K* kernel) {
    cudaFuncAttributes attr;
    return cudaFuncGetAttributes(&attr, reinterpret_cast<const void*>(kernel)) == cudaSuccess;
}

template <int MM>
bool load_dense_kernels() {
    if constexpr (MM >= 4)
        return load_kernel(b200::dense_first_mma_kernel<MM>) && load_kernel(b200::dense_small_mma_kernel<MM>) && load_kernel(b200::dense_dx_mma_kernel<MM>) && load_kernel(b200::dense_wgrad_mma_kernel<MM>);
    else
        return load_kernel(b200::dense_forward_kernel<MM>) && load_kernel(b200::dense_dx_kernel<MM>) && load_kernel(b200::dense_wgrad_kernel<MM>);
}

// The forms of the feature transformer's kernels that a network's kind takes, whatever its batches: each(kernel, has dynamic shared memory).
template <bool PW, bool ONE, class Each>
void each_ft_form_of(bool tiled, Each& each) {
    each(b200::ft_backward_gather_kernel<PW, ONE>, false);
    if (!tiled) return;
    each(b200::ft_forward_tiled_kernel<PW, true>, true), each(b200::ft_forward_tiled_kernel<PW, false>, true);
    each(b200::ft_backward_tiled_kernel<PW, 1024, true, ONE>, true), each(b200::ft_backward_tiled_kernel<PW, 1024, false, ONE>, true);
    each(b200::ft_backward_tiled_kernel<PW, 512, true, ONE>, true), each(b200::ft_backward_tiled_kernel<PW, 512, false, ONE>, true);
    each(b200::ft_csr_kernel, true);
}
template <class Each>
void each_ft_form(const b200_net* net, Each each) {
    const bool one = net->dense_one();
    if (net->d.pairwise) one ? each_ft_form_of<true, true>(net->tiled_ok, each) : each_ft_form_of<true, false>(net->tiled_ok, each);
    else one ? each_ft_form_of<false, true>(net->tiled_ok, each) : each_ft_form_of<false, false>(net->tiled_ok, each);
}

int preload_kernels(b200_net* net) {
    bool ok = true;
    DISPATCH_M(net->d.dense_out[0], ok = load_dense_kernels<MM>());
    ok = ok && load_kernel(b200::dense_regroup_kernel) && load_kernel(dense_one_form(net, false)) && (!net->small_table() || load_kernel(dense_one_form(net, true))) && load_kernel(b200::dense_one_dx_kernel) && load_kernel(b200::copy_outputs_kernel) && load_kernel(b200::dense_fragments_kernel) && load_kernel(b200::dense_small_grads_kernel);
    for (const b200::GatherShape& g : {b200::GatherShape{1, 4, 0, 0}, b200::GatherShape{1, 2, 0, 0}, b200::GatherShape{2, 1, 0, 0}, b200::GatherShape{4, 1, 0, 0}}) {
        ok = ok && load_kernel(net->d.pairwise ? b200::gather_form<true, false>(g) : b200::gather_form<false, false>(g));
        if (net->d.factoriser_rows) ok = ok && load_kernel(net->d.pairwise ? b200::gather_form<true, true>(g) : b200::gather_form<false, true>(g));
    }
    each_ft_form(net, [&](auto* kernel, bool) { ok = ok && load_kernel(kernel); });
    if (net->small_table()) ok = ok && load_kernel(b200::ft_onehot_kernel) && load_kernel(ft_backward_mma(net));
    ok = ok && load_kernel(b200::factoriser_merge_kernel) && load_kernel(b200::factoriser_grad_kernel);
    ok = ok && load_kernel(b200::adamw_flat_kernel) && load_kernel(b200::step_update_kernel) && load_kernel(b200::step_update_copies_kernel<true>) && load_kernel(b200::step_update_copies_kernel<false>) && load_kernel(b200::lookahead_kernel);
    ok = ok && load_kernel(b200::adamw_exchange_kernel<0>) && load_kernel(b200::adamw_exchange_kernel<2>);
    ok = ok && load_kernel(b200::adamw_exchange_kernel<4>) && load_kernel(b200::adamw_exchange_kernel<8>);
    ok = ok && load_kernel(b200::adamw_exchange_bulk_kernel<2, 256, 6>) && load_kernel(b200::adamw_exchange_bulk_kernel<2, 512, 3>);
    ok = ok && load_kernel(b200::adamw_exchange_bulk_kernel<2, 128, 12>) && load_kernel(b200::adamw_exchange_bulk_kernel<4, 256, 5>);
    ok = ok && load_kernel(b200::adamw_exchange_bulk_kernel<0, 256, 3>) && load_kernel(b200::adamw_exchange_bulk_kernel<0, 512, 1>);
    ok = ok && load_kernel(b200::adamw_exchange_bulk_kernel<0, 128, 6>);
    ok = ok && load_kernel(b200::adamw_exchange_overlap_kernel<0>) && load_kernel(b200::adamw_exchange_overlap_kernel<2>);
    ok = ok && load_kernel(b200::adamw_exchange_overlap_kernel<4>) && load_kernel(b200::adamw_exchange_overlap_kernel<8>);
    ok = ok && load_kernel(b200::prep_featurise_kernel) && load_kernel(b200::group_lists_kernel) && load_kernel(b200::group_scan_kernel) && load_kernel(b200::group_place_kernel);
    ok = ok && load_kernel(b200::group_many_count_kernel) && load_kernel(b200::group_many_scan_kernel) && load_kernel(b200::group_many_place_kernel);
    ok = ok && load_kernel(b200::peer_signal_kernel) && load_kernel(b200::peer_wait_kernel) && load_kernel(b200::bucket_presignal_kernel);
    if (!ok) return b200::fail(B200_ERR_CUDA, "net_create: loading the kernels failed: %s", cudaGetErrorString(cudaGetLastError()));
    return 0;
}

}  // namespace

extern "C" {

const char* b200_last_error(void) { return b200::error_buffer(); }
int b200_version(void) { return 1; }

int b200_net_create(int device, void* stream, const b200_net_desc* desc, b200_net** out) {
    if (!desc || !out) return b200::fail(B200_ERR_ARG, "net_create: null argument");
    *out = nullptr;
    if (int rc = validate(*desc)) return rc;
    int count = 0;
    CK(cudaGetDeviceCount(&count));
    if (device < 0 || device >= count) return b200::fail(B200_ERR_CUDA, "net_create: no CUDA device %d (%d visible)", device, count);
    b200_net* net = new b200_net();
    net->device = device;
    net->d = *desc;
    const b200_net_desc& d = net->d;
    auto bail = [&](int rc) {
        b200_net_destroy(net);
        return rc;
    };
    if (int rc = set_device(net)) return bail(rc);
    if (cudaDeviceGetAttribute(&net->sm_count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || net->sm_count < 1)
        return bail(b200::fail(B200_ERR_CUDA, "net_create: cannot read the SM count of device %d", device));
    if (stream) {
        net->stream = static_cast<cudaStream_t>(stream);
    } else {
        if (cudaStreamCreateWithFlags(&net->stream, cudaStreamNonBlocking) != cudaSuccess)
            return bail(b200::fail(B200_ERR_CUDA, "net_create: cannot create a stream"));
        net->own_stream = true;
    }
    if (cudaStreamCreateWithFlags(&net->zero_stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreateWithFlags(&net->zero_fork, cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&net->zero_done, cudaEventDisableTiming) != cudaSuccess)
        return bail(b200::fail(B200_ERR_CUDA, "net_create: cannot create the side stream"));
    if (cudaStreamCreateWithFlags(&net->copy_stream, cudaStreamNonBlocking) != cudaSuccess)
        return bail(b200::fail(B200_ERR_CUDA, "net_create: cannot create the copy stream"));
    {
        int least = 0, greatest = 0;
        cudaDeviceGetStreamPriorityRange(&least, &greatest);
        if (cudaStreamCreateWithPriority(&net->xch_stream, cudaStreamNonBlocking, greatest) != cudaSuccess ||
            cudaEventCreateWithFlags(&net->xch_fork, cudaEventDisableTiming) != cudaSuccess ||
            cudaEventCreateWithFlags(&net->xch_join, cudaEventDisableTiming) != cudaSuccess)
            return bail(b200::fail(B200_ERR_CUDA, "net_create: cannot create the exchange stream"));
    }

    // flat layout, tensors in name order
    auto add = [&](const char* name, int64_t rows, int64_t cols) {
        Tensor t;
        t.name = name;
        t.rows = rows;
        t.cols = cols;
        t.n = rows * cols;
        net->tensors.push_back(t);
    };
    add("l0b", d.ft_out, 1);
    if (d.factoriser_rows) add("l0f", d.ft_out, d.factoriser_rows);
    for (int l = 0; l < d.n_dense; l++) {
        char name[16];
        const int64_t rows = (int64_t)d.n_out_buckets * d.dense_out[l];
        snprintf(name, sizeof name, "l%db", l + 1);
        add(name, rows, 1);
        snprintf(name, sizeof name, "l%dw", l + 1);
        add(name, rows, net->dense_in(l));
    }
    add("l0w", d.ft_out, d.n_inputs);  // last, so that everything else is one contiguous head
    int64_t off = kAlignFloats;                  // float 0 of G is the loss
    for (auto& t : net->tensors) {
        t.off = off;
        off += (t.n + kAlignFloats - 1) / kAlignFloats * kAlignFloats;
    }
    net->n_flat = (off + 1023) / 1024 * 1024;  // a multiple of 4 floats x 256: splits evenly over up to 256 ranks

    constexpr size_t kMaxSmem = 227 * 1024 - 128;  // (the tiled backward's own few bytes count as 128)
    // The tiled kernels need features of one perspective that fall into one block.  A table that is small enough is one block
    // whatever was promised, and then any width will do (a width that 64 does not divide costs as much as the next that does).
    const bool promised = d.ft_block_rows > 0 && d.n_inputs % d.ft_block_rows == 0 && d.ft_out % b200::kTileCols == 0;
    const int R = promised ? d.ft_block_rows : d.n_inputs;
    net->tiled_ok = (promised || (d.pairwise ? d.ft_out / 2 : d.ft_out) >= 32) && R < 1024 &&
                    b200::ft_fwd_fits(R, (d.nnz + 7) & ~7) &&
                    b200::ft_bwd_smem(R, d.nnz, 256) <= kMaxSmem;
    net->tiled_promised = net->tiled_ok && promised;
    net->block_rows = R;
    if (net->tiled_ok)
        for (net->wide_chunk = b200::kChunkMost; b200::ft_bwd_smem(R, d.nnz, net->wide_chunk) > kMaxSmem;) net->wide_chunk -= 8;
    net->nblocks = net->tiled_ok ? d.n_inputs / R : 1;
    net->nslabs = (d.ft_out + b200::kTileCols - 1) / b200::kTileCols;

    const size_t B = d.max_batch;
    for (auto& s : net->slots) {
        slot_layout(net, s, d.max_batch);
        s.n = 0;
    }
    // One allocation for everything but the buffers that peers map: allocations cost a few hundred us each
    Plan plan;
    int rc = 0;
    rc = rc ? rc : dev_alloc(net, &net->P, net->n_flat);
    rc = rc ? rc : dev_alloc(net, &net->G, net->n_flat);
    plan.add(&net->M, net->n_flat);
    plan.add(&net->V, net->n_flat);
    if (d.factoriser_rows) plan.add(&net->table, (size_t)d.n_inputs * d.ft_out);
    plan.add(&net->x, B * net->D1());
    if (d.pairwise) plan.add(&net->u, B * 2 * d.ft_out);
    plan.add(&net->dx, B * net->D1());
    plan.add(&net->a1, B * d.dense_out[0]);
    plan.add(&net->a2, B * 32);
    for (int l = 0; l < 3; l++) plan.add(&net->dz[l], B * 32);
    plan.add(&net->out, B);
    plan.add(&net->d_stamps, b200_net::kTimingRing * b200_net::kTimingEvents);
    plan.add(&net->d_status, b200_net::kLossRing);
    if (net->small_table()) plan.add(&net->gmax, 2);
    if (net->dense_mma()) {
        const size_t table = b200::mma_table_words(net->D1(), d.n_out_buckets, d.dense_out[0]);
        plan.add(&net->w1f, table);
        plan.add(&net->w1d, table);
        // one part per slice, or more of them for few tiles (dense_split)
        const size_t tiles = (size_t)d.max_batch / b200::kDenseTile + std::min(d.n_out_buckets, d.max_batch) + 1;
        plan.add(&net->dz_frag, tiles * (b200::kDenseTile / b200::kWgradStep) * b200::wgrad_table_words<16>(1) * (d.dense_out[0] > 16 ? d.dense_out[0] / 16 : 1));
        plan.add(&net->dense_partial, std::max(dense_slices(net) * tiles, (size_t)8 * net->sm_count) * b200::kDenseTile * d.dense_out[0]);
    } else {
        plan.add(&net->w1g, (size_t)2 * d.n_out_buckets * d.dense_out[0] * net->D1());
        if (net->dense_one()) plan.add(&net->kept_bucket, B);
    }
    // the fence counters get an allocation of their own size class (2 MiB), so that its IPC handle maps exactly it
    rc = rc ? rc : dev_alloc(net, &net->xch_flags, (size_t)(2 << 20) / sizeof(int));
    if (!rc) cudaMemsetAsync(net->xch_flags, 0, (size_t)2 << 20, net->stream);
    plan.add(&net->d_win_rate, 65536);
    plan.add(&net->d_expanded, 64);
    plan.add(&net->d_peers, 1);
    plan.add(&net->done_count, (size_t)net->nblocks);
    if (net->tiled_promised && d.factoriser_rows == d.ft_block_rows)
        plan.add(&net->facc, (size_t)d.ft_block_rows * d.ft_out / 2);
    if (net->tiled_ok) {
        // sized for whichever chunk length needs most, of all that bwd_chunk may choose for a batch: how many chunks there can be
        // falls in steps, so a length in between may need more than the shortest and the longest
        size_t ent_total = 0, start_total = 0;
        auto room_for = [&](int cp) {
            const size_t chunks = most_chunks(net, (int)B, cp);
            start_total = std::max(start_total, chunks * b200::ft_bwd_start_cap(R, d.nnz, cp));
            ent_total = std::max(ent_total, chunks * b200::ft_bwd_ent_cap(R, d.nnz, cp));
        };
        room_for(b200::ft_bwd_chunk_narrow(d.nnz));
        for (int cp = net->wide_chunk; cp >= b200::kChunkLeast; cp -= 8) room_for(cp);
        room_for(net->wide_chunk);
        if (R < b200::kMmaTileRows) {
            const size_t steps = most_chunks(net, (int)B, b200::kStepPairs);
            start_total = std::max(start_total, steps * b200::kStepHead);
            ent_total = std::max(ent_total, steps * b200::ft_mma_ent_cap(R));
        }
        for (auto& s : net->slots) {
            plan.add(&s.lists, 2 * B * ((d.nnz + 7) & ~7));
            plan.add(&s.csr_ent, ent_total);
            plan.add(&s.csr_start, start_total);
        }
    }
    for (auto& s : net->slots) plan.add(&s.d_blob, s.bytes);
    rc = rc ? rc : plan.allocate(net);
    if (!rc) cudaMemsetAsync(net->done_count, 0, (size_t)net->nblocks * sizeof(int), net->stream);
    if (rc) return bail(rc);
    if (!d.factoriser_rows) net->table = net->P + net->find("l0w")->off;
    cudaMemsetAsync(net->P, 0, net->n_flat * 4, net->stream);
    cudaMemsetAsync(net->G, 0, net->n_flat * 4, net->stream);
    cudaMemsetAsync(net->M, 0, net->n_flat * 4, net->stream);
    cudaMemsetAsync(net->V, 0, net->n_flat * 4, net->stream);

    const size_t pinned_slot = align_up(std::max(net->slots[0].off_records, (size_t)d.max_batch * 36), 4096);
    {   // pinned memory: the slots' staging blocks, the outputs of an evaluation, the read-back ring
        void* raw = nullptr;
        const size_t out_bytes = align_up(B * sizeof(float), 4096);
        if (cudaHostAlloc(&raw, B200_NUM_SLOTS * pinned_slot + out_bytes + 128, cudaHostAllocDefault) != cudaSuccess)
            return bail(b200::fail(B200_ERR_CUDA, "net_create: pinned allocation failed"));
        net->h_pinned = static_cast<char*>(raw);
        net->h_out = reinterpret_cast<float*>(net->h_pinned + B200_NUM_SLOTS * pinned_slot);
        net->h_loss = reinterpret_cast<float*>(net->h_pinned + B200_NUM_SLOTS * pinned_slot + out_bytes);
    }
    for (auto& s : net->slots) {
        s.h_blob = net->h_pinned + (&s - net->slots) * pinned_slot;
        cudaEventCreateWithFlags(&s.ready, cudaEventDisableTiming);
        cudaEventCreateWithFlags(&s.consumed, cudaEventDisableTiming);
        s.n = 0;
    }
    net->h_status = reinterpret_cast<int*>(net->h_loss + 8);
    net->h_xstatus = net->h_status + b200_net::kLossRing;
    net->h_gave_up = net->h_xstatus + 4 * b200_net::kLossRing;
    memset(net->h_loss, 0, 128);  // 8 floats, 4 status words, 4 x 4 fence words, the wait word
    for (auto& e : net->loss_ev) cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
    {
        auto set_dense = [&](int m) -> int {
            cudaError_t e = cudaSuccess;
            DISPATCH_M(m, e = set_dense_forward_smem<MM>());
            if (e != cudaSuccess) return b200::fail(B200_ERR_CUDA, "dense forward shared memory: %s", cudaGetErrorString(e));
            return 0;
        };
        if (int rc2 = set_dense(d.dense_out[0])) return bail(rc2);
        if (b200::allow_smem(dense_one_form(net, false)) != cudaSuccess || (net->small_table() && b200::allow_smem(dense_one_form(net, true)) != cudaSuccess)) return bail(b200::fail(B200_ERR_CUDA, "net_create: shared memory of the dense kernel"));
    }
    if (net->tiled_ok) {
        cudaError_t e = cudaSuccess;
        each_ft_form(net, [&](auto* kernel, bool dynamic) {
            if (dynamic && e == cudaSuccess) e = b200::allow_smem(kernel);
        });
        if (net->small_table()) e = e ? e : b200::allow_smem(ft_backward_mma(net));
        if (e != cudaSuccess) return bail(b200::fail(B200_ERR_CUDA, "net_create: shared memory of the tiled kernels: %s", cudaGetErrorString(e)));
    }
    cudaFuncSetAttribute(b200::adamw_exchange_overlap_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, b200::kOverlapSmem);
    cudaFuncSetAttribute(b200::adamw_exchange_overlap_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, b200::kOverlapSmem);
    cudaFuncSetAttribute(b200::adamw_exchange_overlap_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, b200::kOverlapSmem);
    cudaFuncSetAttribute(b200::adamw_exchange_overlap_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, b200::kOverlapSmem);
    if (int rc2 = preload_kernels(net)) return bail(rc2);
    CK(cudaStreamSynchronize(net->stream));
    CK(cudaGetLastError());
    *out = net;
    return 0;
}

int b200_net_destroy(b200_net* net) {
    if (!net) return 0;
    cudaSetDevice(net->device);
    if (net->stream) cudaStreamSynchronize(net->stream);
    if (net->copy_stream) cudaStreamSynchronize(net->copy_stream);
    if (net->zero_stream) cudaStreamSynchronize(net->zero_stream);
    if (net->xch_stream) cudaStreamSynchronize(net->xch_stream);
    for (int r = 0; r < net->xch_world; r++)
        if (r != net->xch_rank) {
            if (net->peer_g[r]) cudaIpcCloseMemHandle(net->peer_g[r]);
            if (net->peer_p[r]) cudaIpcCloseMemHandle(net->peer_p[r]);
            if (net->peer_flags[r]) cudaIpcCloseMemHandle(net->peer_flags[r]);
        }
    for (void* p : net->allocations) cudaFree(p);
    for (auto& s : net->slots) {
        if (s.ready) cudaEventDestroy(s.ready);
        if (s.consumed) cudaEventDestroy(s.consumed);
    }
    if (net->h_pinned) cudaFreeHost(net->h_pinned);
    for (auto& e : net->loss_ev)
        if (e) cudaEventDestroy(e);
    for (auto& ring : net->tev)
        for (auto& e : ring)
            if (e) cudaEventDestroy(e);
    if (net->own_stream && net->stream) cudaStreamDestroy(net->stream);
    if (net->copy_stream) cudaStreamDestroy(net->copy_stream);
    if (net->zero_stream) cudaStreamDestroy(net->zero_stream);
    if (net->xch_stream) cudaStreamDestroy(net->xch_stream);
    if (net->xch_fork) cudaEventDestroy(net->xch_fork);
    if (net->xch_join) cudaEventDestroy(net->xch_join);
    if (net->zero_fork) cudaEventDestroy(net->zero_fork);
    if (net->zero_done) cudaEventDestroy(net->zero_done);
    delete net;
    return 0;
}

int b200_net_set_option(b200_net* net, const char* key, int64_t value) {
    if (!net || !key) return b200::fail(B200_ERR_ARG, "set_option: null argument");
    if (!strcmp(key, "ft_mode") || !strcmp(key, "ft_fwd_mode") || !strcmp(key, "ft_bwd_mode")) {
        if (value < B200_FT_AUTO || value > B200_FT_TILED) return b200::fail(B200_ERR_ARG, "ft_mode %lld unknown", (long long)value);
        if (value == B200_FT_TILED && !net->tiled_promised)
            return b200::fail(B200_ERR_UNSUPPORTED,
                              "tiled feature-transformer kernels need ft_block_rows > 0 dividing n_inputs, at most "
                              "about 800 rows per block, and ft_out a multiple of 64");
        if (strcmp(key, "ft_bwd_mode")) net->ft_fwd_mode = (int)value;
        if (strcmp(key, "ft_fwd_mode")) net->ft_bwd_mode = (int)value;
        return 0;
    }
    if (!strcmp(key, "exchange_wait_ms")) {  // how long a fence of the peer exchange polls before it gives up
        net->xch_spin_limit = std::max<int64_t>(1, value) * 5000;
        return 0;
    }
    if (!strcmp(key, "exchange_ctas")) {
        net->exchange_ctas = (int)std::max<int64_t>(0, value);
        return 0;
    }
    if (!strcmp(key, "overlap_ctas")) {  // SMs that b200_step_exchange takes away from the backward for the exchange
        if (value < 1 || value >= net->sm_count) return b200::fail(B200_ERR_ARG, "overlap_ctas must be in [1, %d)", net->sm_count);
        net->overlap_ctas = (int)value;
        return 0;
    }
    if (!strcmp(key, "overlap_mode")) {  // takes effect for batches uploaded afterwards
        net->overlap_mode = value != 0;
        return 0;
    }
    if (!strcmp(key, "exchange_step")) {
        // After a step that reported B200_ERR_STATE the ranks' step counters may differ.  Every rank, with nothing
        // in flight and after a host-side barrier, sets the same value, larger than any count reached so far;
        // the call also clears this rank's timeout word.
        if (value < net->xch_step) return b200::fail(B200_ERR_ARG, "exchange_step must not go back (now %d)", net->xch_step);
        if (int rc = set_device(net)) return rc;
        CK(cudaStreamSynchronize(net->stream));
        CK(cudaStreamSynchronize(net->xch_stream));
        CK(cudaMemset(net->xch_flags + b200::kFlagTimeout, 0, 4 * sizeof(int)));
        CK(cudaMemset(net->done_count, 0, (size_t)net->nblocks * sizeof(int)));
        net->xch_step = (int)value;
        return 0;
    }
    if (!strcmp(key, "manual_grad_zero")) {
        net->manual_grad_zero = value != 0;
        return 0;
    }
    if (!strcmp(key, "exchange_bulk")) {  // 0: the exchange kernel fetches peer gradients with per-thread loads
        net->exchange_bulk = (int)value;
        return 0;
    }
    if (!strcmp(key, "ft_bwd_grab")) {
        if (value < 0 || value > 64) return b200::fail(B200_ERR_ARG, "ft_bwd_grab must be in [0, 64]");
        return 0;  // (all pieces are dealt out in advance)
    }
    if (!strcmp(key, "ft_once")) {
        return 0;  // (no load of the tiled kernels gains from an L1 line any more: one form)
    }
    if (!strcmp(key, "ft_bwd_products")) {  // takes effect for batches uploaded afterwards
        if (value < -1 || value > 1) return b200::fail(B200_ERR_ARG, "ft_bwd_products must be -1, 0 or 1");
        net->bwd_products = (int)value;
        return 0;
    }
    if (!strcmp(key, "ft_bwd_wide")) {  // takes effect for batches uploaded afterwards
        net->bwd_wide = value != 0;
        return 0;
    }
    return b200::fail(B200_ERR_ARG, "set_option: unknown key '%s'", key);
}

int b200_net_tensor_size(b200_net* net, const char* name, int64_t* n) {
    if (!net || !name || !n) return b200::fail(B200_ERR_ARG, "tensor_size: null argument");
    const Tensor* t = net->find(name);
    if (!t) return b200::fail(B200_ERR_ARG, "no tensor named '%s' in this network", name);
    *n = t->n;
    return 0;
}

int b200_net_tensor_offset(b200_net* net, const char* name, int64_t* first_float) {
    if (!net || !name || !first_float) return b200::fail(B200_ERR_ARG, "tensor_offset: null argument");
    const Tensor* t = net->find(name);
    if (!t) return b200::fail(B200_ERR_ARG, "no tensor named '%s' in this network", name);
    *first_float = t->off;
    return 0;
}

int b200_net_tensor_shape(b200_net* net, const char* name, int64_t* rows, int64_t* cols) {
    if (!net || !name || !rows || !cols) return b200::fail(B200_ERR_ARG, "tensor_shape: null argument");
    const Tensor* t = net->find(name);
    if (!t) return b200::fail(B200_ERR_ARG, "no tensor named '%s' in this network", name);
    *rows = t->rows;
    *cols = t->cols;
    return 0;
}

static float* kind_base(b200_net* net, int kind) {
    switch (kind) {
        case B200_KIND_WEIGHT: return net->P;
        case B200_KIND_MOMENTUM: return net->M;
        case B200_KIND_VELOCITY: return net->V;
        case B200_KIND_GRAD: return net->G;
        case B200_KIND_SLOW: return net->S;
        default: return nullptr;
    }
}

int b200_net_set_tensor(b200_net* net, const char* name, int kind, const float* host, int64_t n) {
    if (!net || !name || !host) return b200::fail(B200_ERR_ARG, "set_tensor: null argument");
    const Tensor* t = net->find(name);
    if (!t) return b200::fail(B200_ERR_ARG, "no tensor named '%s' in this network", name);
    if (n != t->n) return b200::fail(B200_ERR_ARG, "tensor '%s' holds %lld values, %lld given", name, (long long)t->n, (long long)n);
    if ((kind < B200_KIND_WEIGHT || kind > B200_KIND_VELOCITY) && kind != B200_KIND_SLOW)
        return b200::fail(B200_ERR_ARG, "set_tensor: kind %d is not writable", kind);
    if (kind == B200_KIND_SLOW && !net->S) return b200::fail(B200_ERR_STATE, "set_tensor: no tensor of this network uses Ranger");
    if (int rc = set_device(net)) return rc;
    CK(cudaStreamSynchronize(net->stream));
    CK(cudaMemcpy(kind_base(net, kind) + t->off, host, n * sizeof(float), cudaMemcpyHostToDevice));
    if (kind == B200_KIND_WEIGHT) net->weights_moved();
    return 0;
}

int b200_net_get_tensor(b200_net* net, const char* name, int kind, float* host, int64_t n) {
    if (!net || !name || !host) return b200::fail(B200_ERR_ARG, "get_tensor: null argument");
    const Tensor* t = net->find(name);
    if (!t) return b200::fail(B200_ERR_ARG, "no tensor named '%s' in this network", name);
    if (n != t->n) return b200::fail(B200_ERR_ARG, "tensor '%s' holds %lld values, %lld asked", name, (long long)t->n, (long long)n);
    float* base = kind_base(net, kind);
    if (!base) return b200::fail(B200_ERR_ARG, "get_tensor: unknown kind %d (or no tensor uses Ranger's slow weights)", kind);
    if (int rc = set_device(net)) return rc;
    CK(cudaStreamSynchronize(net->stream));
    CK(cudaMemcpy(host, base + t->off, n * sizeof(float), cudaMemcpyDeviceToHost));
    return 0;
}

int b200_net_set_adamw(b200_net* net, const char* name, const b200_adamw_params* params) {
    if (!net || !params) return b200::fail(B200_ERR_ARG, "set_adamw: null argument");
    if (!(params->min_weight <= params->max_weight)) return b200::fail(B200_ERR_ARG, "set_adamw: min_weight > max_weight");
    if (!name) {
        for (auto& t : net->tensors) t.hp = *params, t.opt_kind = B200_OPT_ADAMW;
        return 0;
    }
    Tensor* t = net->find(name);
    if (!t) return b200::fail(B200_ERR_ARG, "no tensor named '%s' in this network", name);
    t->hp = *params;
    t->opt_kind = B200_OPT_ADAMW;
    return 0;
}

int b200_net_set_optimiser(b200_net* net, const char* name, const b200_optimiser_params* params) {
    if (!net || !params) return b200::fail(B200_ERR_ARG, "set_optimiser: null argument");
    if (params->kind < B200_OPT_ADAMW || params->kind > B200_OPT_RANGER) return b200::fail(B200_ERR_ARG, "set_optimiser: unknown kind %d", params->kind);
    if (!(params->min_weight <= params->max_weight)) return b200::fail(B200_ERR_ARG, "set_optimiser: min_weight > max_weight");
    if (params->kind == B200_OPT_RANGER && (params->k < 1 || !(params->alpha >= 0.f && params->alpha <= 1.f)))
        return b200::fail(B200_ERR_ARG, "set_optimiser: Ranger needs k >= 1 and alpha in [0, 1]");
    Tensor* only = nullptr;
    if (name && !(only = net->find(name))) return b200::fail(B200_ERR_ARG, "no tensor named '%s' in this network", name);
    if (int rc = set_device(net)) return rc;
    if (params->kind == B200_OPT_RANGER && !net->S) {  // slow weights start at zero, as in the reference (ranger.rs:70)
        if (int rc = dev_alloc(net, &net->S, (size_t)net->n_flat)) return rc;
        CK(cudaMemset(net->S, 0, (size_t)net->n_flat * sizeof(float)));
    }
    for (auto& t : net->tensors) {
        if (only && &t != only) continue;
        t.hp = {params->decay, params->beta1, params->beta2, params->min_weight, params->max_weight};
        t.opt_kind = params->kind;
        t.n_sma_threshold = params->n_sma_threshold;
        t.alpha = params->alpha;
        t.lookahead_k = params->k;
    }
    net->opt_step = 0;  // OptimiserState::set_params of the lookahead resets its step (ranger.rs:107-113)
    return 0;
}

// Common start of both uploads: the slot's pinned block is free once its last copy has landed and
// the last step that read the device block has finished.
static int upload_begin(b200_net* net, int slot, int32_t n, const char* who) {
    if (slot < 0 || slot >= B200_NUM_SLOTS) return b200::fail(B200_ERR_ARG, "%s: slot %d out of range", who, slot);
    if (n < 1 || n > net->d.max_batch) return b200::fail(B200_ERR_ARG, "%s: %d positions, capacity is %d", who, n, net->d.max_batch);
    if (int rc = set_device(net)) return rc;
    Slot& s = net->slots[slot];
    if (s.has_ready) CK(cudaEventSynchronize(s.ready));
    if (s.has_consumed) CK(cudaEventSynchronize(s.consumed));
    slot_layout(net, s, n);
    s.n = 0;
    return 0;
}

// The row lists of the tiled kernels depend on the indices only: they are built right behind the copy, on the copy stream,
// where they run beside the step that is still computing.  What only the backward reads waits for a network that trains.
static bool upload_wants_lists(const b200_net* net, int32_t n) {
    return net->tiled_ok && (net->trains ? net->fwd_tiled() || net->bwd_tiled() : net->fwd_tiled(n));
}

// Common end: the slot's batch is on its way to the device; group it and mark the slot ready.
static int upload_finish(b200_net* net, Slot& s, bool want_order, bool counted) {
    const bool want_lists = upload_wants_lists(net, s.n);
    if (want_lists || want_order)
        if (int rc = group_slot(net, s, group_args(net, s, want_lists, want_order), counted, net->copy_stream)) return rc;
    if (want_lists && net->bwd_tiled() && net->trains)
        if (int rc = build_csr(net, s, net->copy_stream)) return rc;
    CK(cudaEventRecord(s.ready, net->copy_stream));
    s.has_ready = true;
    s.has_consumed = false;
    return 0;
}

int b200_batch_upload(b200_net* net, int slot, const int32_t* stm, const int32_t* nstm, const int32_t* buckets,
                      const float* targets, int32_t n) {
    if (!net || !stm || !nstm || !targets) return b200::fail(B200_ERR_ARG, "batch_upload: null argument");
    const b200_net_desc& d = net->d;
    if (d.n_out_buckets > 1 && !buckets) return b200::fail(B200_ERR_ARG, "batch_upload: this network needs output buckets");
    if (int rc = upload_begin(net, slot, n, "batch_upload")) return rc;
    Slot& s = net->slots[slot];
    const int64_t count = (int64_t)n * d.nnz;
    uint16_t* h_stm = s.host<uint16_t>(s.off_stm);
    uint16_t* h_nstm = s.host<uint16_t>(s.off_nstm);
    const uint32_t limit = (uint32_t)d.n_inputs;
#pragma omp parallel for schedule(static) if (count > 200000)
    for (int64_t i = 0; i < count; i++) {
        const uint32_t a = (uint32_t)stm[i], b = (uint32_t)nstm[i];
        h_stm[i] = a < limit ? (uint16_t)a : (uint16_t)0xFFFFu;
        h_nstm[i] = b < limit ? (uint16_t)b : (uint16_t)0xFFFFu;
    }
    int* h_buckets = s.host<int>(s.off_buckets);
    const int O = d.n_out_buckets;
    if (buckets) {
        for (int i = 0; i < n; i++) {
            if ((unsigned)buckets[i] >= (unsigned)O)
                return b200::fail(B200_ERR_DATA, "batch_upload: position %d has output bucket %d, network has %d", i, buckets[i], O);
            h_buckets[i] = buckets[i];
        }
    } else {
        memset(h_buckets, 0, (size_t)n * 4);
    }
    memcpy(s.host<float>(s.off_targets), targets, (size_t)n * 4);
    s.n = n;
    s.prepared = s.csr_built = false;
    cut_dense(net, s);
    cut_ft(net, s);
    // positions by output bucket: with the row lists on the device; for a batch that needs no lists here, which is a small
    // one or one of a network without them, before the copy: two launches fewer
    const bool order_here = O > 1 && !upload_wants_lists(net, n) && n <= 4096;
    size_t bytes = s.off_order;
    if (order_here) {
        int begin[b200::kGroupMaxBuckets + 1] = {0};
        for (int i = 0; i < n; i++) begin[h_buckets[i] + 1]++;
        int2* h_tiles = s.host<int2>(s.off_dtiles);
        s.n_dtiles = 0;
        for (int k = 0; k < O; k++) {
            begin[k + 1] += begin[k];
            for (int at = begin[k]; at < begin[k + 1]; at += b200::kDenseTile)
                h_tiles[s.n_dtiles++] = make_int2(at, std::min(b200::kDenseTile, begin[k + 1] - at));
        }
        int* h_order = s.host<int>(s.off_order);
        for (int i = 0; i < n; i++) h_order[begin[h_buckets[i]]++] = i;
        bytes = s.off_records;
    }
    CK(cudaMemcpyAsync(s.d_blob, s.h_blob, bytes, cudaMemcpyHostToDevice, net->copy_stream));
    net->h2d_bytes += (int64_t)bytes;
    return upload_finish(net, s, O > 1 && !order_here, false);
}

// Records in, batch prepared on the device: the raw 32 bytes per position are checked while they are copied into the
// pinned block and cross PCIe as they are; the featuriser, the output bucket and the target blend of
// ValueTrainerState::make_mapper (crates/bullet_lib/src/value.rs:77-117) and the grouping run as kernels on the copy
// stream.  Nothing is read back, so the call returns when everything is enqueued.
static int upload_records(b200_net* net, int slot, const void* records, int32_t n, int32_t game, const int32_t* layout32, float scale, float blend,
                          const char* who) {
    if (!net || !records) return b200::fail(B200_ERR_ARG, "%s: null argument", who);
    if (game < B200_GAME_CHESS768 || game > B200_GAME_ATAXX147) return b200::fail(B200_ERR_ARG, "%s: unknown game %d", who, game);
    if (game == B200_GAME_CHESS_BUCKETS_MIRRORED && !layout32) return b200::fail(B200_ERR_ARG, "%s: the king-bucket layout is missing", who);
    if (!(blend >= 0.f && blend <= 1.f) || !(scale > 0.f)) return b200::fail(B200_ERR_ARG, "%s: bad scale or blend", who);
    const b200_net_desc& d = net->d;
    const int O = d.n_out_buckets;
    if (O > 1 && game == B200_GAME_ATAXX147) return b200::fail(B200_ERR_UNSUPPORTED, "%s: no output buckets for ataxx records", who);
    if (int rc = upload_begin(net, slot, n, who)) return rc;
    Slot& s = net->slots[slot];
    // The device looks the win rate of a score up in a table, which takes the host as long to make as the targets of 65536
    // positions do: until a scale has seen that many, the host forms the targets while it goes through the records.
    // (First upload and evaluation of a network, king buckets, width 2048, with the table made first and now: 1 position 357
    // and 120 us, 1024 434 and 197, 16384 696 and 464.)
    bool host_targets = false;
    if (net->win_rate_scale != scale) {
        if (net->host_scale != scale) net->host_scale = scale, net->host_positions = 0;
        net->host_positions += n;
        host_targets = net->host_positions < 65536;
    }
    const float rscale = 1.0f / scale;
    if (net->win_rate_scale != scale && !host_targets) {  // the same function the host mapper evaluates, for every possible score
        std::vector<float> table(65536);
#pragma omp parallel for schedule(static)
        for (int v = -32768; v < 32768; v++) table[v + 32768] = b200::blended_target((int16_t)v, 0, rscale, 0.0f);
        // (behind the kernels that read the table before; out of pageable memory, so it has been read when the call returns)
        CK(cudaMemcpyAsync(net->d_win_rate, table.data(), table.size() * sizeof(float), cudaMemcpyHostToDevice, net->copy_stream));
        net->win_rate_scale = scale;
        net->host_positions = 0;
    }
    if (game == B200_GAME_CHESS_BUCKETS_MIRRORED && (!net->expanded_valid || memcmp(net->expanded_layout, layout32, sizeof net->expanded_layout))) {
        int32_t expanded[64];
        b200::expand_king_buckets(layout32, expanded);
        net->expanded_valid = false;
        CK(cudaMemcpyAsync(net->d_expanded, expanded, sizeof expanded, cudaMemcpyHostToDevice, net->copy_stream));
        memcpy(net->expanded_layout, layout32, sizeof net->expanded_layout);
        net->expanded_valid = true;
    }
    float* targets = reinterpret_cast<float*>(s.h_blob + (size_t)n * 32);  // behind the records
    int bad = n, bad_bucket = n;
    {
        const b200::AtaxxRecord* in = static_cast<const b200::AtaxxRecord*>(records);  // (both kinds start with 64-bit boards)
        b200::AtaxxRecord* out = reinterpret_cast<b200::AtaxxRecord*>(s.h_blob);
        const int nnz = d.nnz;
        const bool ataxx = game == B200_GAME_ATAXX147;
#pragma omp parallel for schedule(static) reduction(min : bad) reduction(min : bad_bucket) if (n >= (host_targets ? 2048 : 8192))
        for (int32_t i = 0; i < n; i++) {
            const b200::AtaxxRecord r = in[i];
            out[i] = r;
            if (host_targets) targets[i] = b200::blended_target(r.score, r.result, rscale, blend);  // same offsets in both record types
            int pieces = __builtin_popcountll(r.bbs[0]);
            if (ataxx) pieces += __builtin_popcountll(r.bbs[1]) + __builtin_popcountll(r.bbs[2]);
            if (pieces > nnz) bad = i < bad ? i : bad;
            if (O > 1 && (unsigned)b200::material_bucket(r.bbs[0], O) >= (unsigned)O) bad_bucket = i < bad_bucket ? i : bad_bucket;
        }
    }
    if (bad < n) return b200::fail(B200_ERR_DATA, "%s: record %d holds more than nnz=%d pieces", who, bad, d.nnz);
    if (bad_bucket < n) return b200::fail(B200_ERR_DATA, "%s: record %d has no valid output bucket", who, bad_bucket);
    const size_t bytes = (size_t)n * (host_targets ? 36 : 32);
    net->h2d_bytes += (int64_t)bytes;
    s.n = n;
    s.prepared = s.csr_built = false;
    cut_dense(net, s);
    cut_ft(net, s);
    b200::PrepArgs p{};
    // an evaluation waits for its batch: the featuriser then reads the pinned block itself.  (Beside a training step its CTAs
    // would wait for PCIe on SMs that the step could use.)
    const bool direct = !net->trains && n <= 16384;
    p.records = direct ? reinterpret_cast<const uint4*>(s.h_blob) : s.dev<uint4>(s.off_records);
    if (host_targets) p.given = reinterpret_cast<const float*>(p.records + 2 * (size_t)n);
    p.game = game;
    p.expanded = net->d_expanded;
    p.win_rate = net->d_win_rate;
    p.blend = blend;
    p.stm = s.dev<uint16_t>(s.off_stm);
    p.nstm = s.dev<uint16_t>(s.off_nstm);
    p.buckets = s.dev<int>(s.off_buckets);
    p.targets = s.dev<float>(s.off_targets);
    if (!direct) CK(cudaMemcpyAsync(s.d_blob + s.off_records, s.h_blob, bytes, cudaMemcpyHostToDevice, net->copy_stream));
    const b200::GroupArgs g = group_args(net, s, upload_wants_lists(net, n), O > 1);
    b200::prep_featurise_kernel<<<b200::group_ctas(n), b200::kPrepThreads, 0, net->copy_stream>>>(p, g);
    LAUNCHED(net);
    return upload_finish(net, s, O > 1, true);
}

int b200_batch_upload_records(b200_net* net, int slot, const void* records, int32_t n, int32_t game, const int32_t* layout32,
                              float scale, float blend) {
    return upload_records(net, slot, records, n, game, layout32, scale, blend, "batch_upload_records");
}
int b200_batch_upload_records_gpu(b200_net* net, int slot, const void* records, int32_t n, int32_t game, const int32_t* layout32,
                                  float scale, float blend) {
    return upload_records(net, slot, records, n, game, layout32, scale, blend, "batch_upload_records_gpu");
}

int b200_slot_read(b200_net* net, int slot, uint16_t* stm, uint16_t* nstm, int32_t* buckets, float* targets, int32_t* order,
                   int32_t* pair_order, int32_t* n) {
    if (int rc = check_slot(net, slot, "slot_read")) return rc;
    if (int rc = set_device(net)) return rc;
    Slot& s = net->slots[slot];
    CK(cudaStreamSynchronize(net->copy_stream));
    const size_t count = (size_t)s.n, list = count * net->d.nnz * sizeof(uint16_t);
    if (stm) CK(cudaMemcpy(stm, s.d_blob + s.off_stm, list, cudaMemcpyDeviceToHost));
    if (nstm) CK(cudaMemcpy(nstm, s.d_blob + s.off_nstm, list, cudaMemcpyDeviceToHost));
    if (buckets) CK(cudaMemcpy(buckets, s.d_blob + s.off_buckets, count * 4, cudaMemcpyDeviceToHost));
    if (targets) CK(cudaMemcpy(targets, s.d_blob + s.off_targets, count * 4, cudaMemcpyDeviceToHost));
    // Both groupings as the kernels have them, every group in ascending order (which the kernels keep for the positions of up to
    // kGroupMaxBlocks row blocks only: they visit the pairs of a block in the order of their lists' lengths).
    if (order && net->d.n_out_buckets > 1) {
        std::vector<int> bucket(count);
        CK(cudaMemcpy(bucket.data(), s.d_blob + s.off_buckets, count * 4, cudaMemcpyDeviceToHost));
        CK(cudaMemcpy(order, s.d_blob + s.off_order, count * 4, cudaMemcpyDeviceToHost));
        if (net->nblocks > b200::kGroupMaxBlocks)
            for (size_t at = 0, end; at < count; at = end) {  // runs of one bucket
                for (end = at + 1; end < count && bucket[order[end]] == bucket[order[at]];) end++;
                std::sort(order + at, order + end);
            }
    } else if (order) {
        for (size_t i = 0; i < count; i++) order[i] = (int32_t)i;
    }
    if (pair_order && net->tiled_ok) {
        if (!s.prepared) {  // (a batch that no tiled kernel has needed yet)
            cut_ft(net, s);
            if (int rc = group_slot(net, s, group_args(net, s, true, false), false, net->copy_stream)) return rc;
            CK(cudaStreamSynchronize(net->copy_stream));
        }
        CK(cudaStreamSynchronize(net->stream));  // (the lists may have been made by a training pass)
        std::vector<int2> pairs(2 * count);
        std::vector<int> begin(net->nblocks + 1);
        CK(cudaMemcpy(pairs.data(), s.d_blob + s.off_pairs, pairs.size() * sizeof(int2), cudaMemcpyDeviceToHost));
        CK(cudaMemcpy(begin.data(), s.d_blob + s.off_blocks, begin.size() * sizeof(int), cudaMemcpyDeviceToHost));
        for (size_t i = 0; i < 2 * count; i++) pair_order[i] = pairs[i].x;
        for (int k = 0; k < net->nblocks; k++) std::sort(pair_order + begin[k], pair_order + begin[k + 1]);
    } else if (pair_order) {  // without row blocks the pairs are visited as they come
        for (size_t i = 0; i < 2 * count; i++) pair_order[i] = (int32_t)i;
    }
    if (n) *n = s.n;
    return 0;
}

// ---- the training forward pass in pieces (b200_backward_begin runs them itself when the caller has not)

// Clears the gradient buffer on a side stream, beside the FT forward, which does not touch it; the dense layers wait for it.
static int clear_gradients_aside(b200_net* net) {
    CK(cudaEventRecord(net->zero_fork, net->stream));
    CK(cudaStreamWaitEvent(net->zero_stream, net->zero_fork, 0));
    CK(cudaMemsetAsync(net->G, 0, (size_t)net->n_flat * 4, net->zero_stream));
    CK(cudaEventRecord(net->zero_done, net->zero_stream));
    net->zero_pending = true;
    return 0;
}

int b200_forward_begin(b200_net* net, int slot) {
    if (int rc = check_slot(net, slot, "forward_begin")) return rc;
    if (net->bwd_slot >= 0) return b200::fail(B200_ERR_STATE, "forward_begin: the backward pass of slot %d is not finished", net->bwd_slot);
    if (int rc = set_device(net)) return rc;
    Slot& s = net->slots[slot];
    CK(cudaStreamWaitEvent(net->stream, s.ready, 0));
    net->trains = true;
    if (int rc = refresh_table(net, s.n)) return rc;
    if (!net->manual_grad_zero) {
        // every gradient is accumulated with reductions, so the buffer starts at zero; nothing before
        // the dense layers writes to it
        if (int rc = clear_gradients_aside(net)) return rc;
    }
    if (!net->events_made) {  // the steps that run in pieces are timed with events
        for (auto& ring : net->tev)
            for (auto& e : ring) CK(cudaEventCreate(&e));
        net->events_made = true;
    }
    net->stamped[net->steps_begun % b200_net::kTimingRing] = false;
    if (int rc = forward_prepare(net, s, true)) return rc;
    net->fwd_slot = slot;
    net->fwd_parts_done = 0;
    net->fwd_parts = 0;
    return 0;
}

int b200_forward_ft(b200_net* net, int slot, int part, int n_parts) {
    if (int rc = check_slot(net, slot, "forward_ft")) return rc;
    if (net->fwd_slot != slot) return b200::fail(B200_ERR_STATE, "forward_ft: call b200_forward_begin on slot %d first", slot);
    if (n_parts < 1 || part < 0 || part >= n_parts || part != net->fwd_parts_done)
        return b200::fail(B200_ERR_ARG, "forward_ft: parts must be run in order 0..n_parts-1 (got %d of %d)", part, n_parts);
    if (n_parts > 1 && (!net->fwd_tiled() || net->nblocks % n_parts))
        return b200::fail(B200_ERR_UNSUPPORTED, "forward_ft: %d parts need the tiled forward and must divide the %d row blocks", n_parts,
                          net->nblocks);
    if (int rc = set_device(net)) return rc;
    Slot& s = net->slots[slot];
    const int per = net->nblocks / n_parts;  // this part's run of row blocks
    if (int rc = forward_ft_blocks(net, s, part * per, n_parts > 1 ? (part + 1) * per : net->nblocks)) return rc;
    net->fwd_parts_done = part + 1;
    net->fwd_parts = n_parts;
    return 0;
}

// ---- the backward pass in three phases (b200_backward runs them back to back)

int b200_backward_begin(b200_net* net, int slot) {
    if (int rc = check_slot(net, slot, "backward_begin")) return rc;
    if (int rc = set_device(net)) return rc;
    Slot& s = net->slots[slot];
    const b200_net_desc& d = net->d;
    if (net->fwd_slot == slot) {  // the forward pass was started in pieces: every piece must be in
        if (net->fwd_parts_done < 1 || net->fwd_parts_done != net->fwd_parts)
            return b200::fail(B200_ERR_STATE, "backward_begin: run every b200_forward_ft part of slot %d first", slot);
    } else {
        if (net->fwd_slot >= 0) return b200::fail(B200_ERR_STATE, "backward_begin: a forward pass of slot %d is under way", net->fwd_slot);
        if (int rc = b200_forward_begin(net, slot)) return rc;
        if (int rc = b200_forward_ft(net, slot, 0, 1)) return rc;
    }
    net->fwd_slot = -1;
    if (int rc = forward_dense(net, s, true)) return rc;
    cudaEvent_t* ev = net->tev[net->steps_begun % b200_net::kTimingRing];
    CK(cudaEventRecord(ev[2], net->stream));
    if (net->bwd_tiled() && !s.csr_built)  // normally built at upload
        if (int rc = build_csr(net, s, net->stream)) return rc;
    if (!net->dense_one()) {
        b200::DenseArgs da = dense_args(net, s, true);
        DISPATCH_M(d.dense_out[0], launch_dense_dx<MM>(net, da, s.n_dtiles));
        LAUNCHED(net);
        if (int rc = launch_dense_grads(net, s)) return rc;
    }
    CK(cudaEventRecord(ev[3], net->stream));
    net->bwd_slot = slot;
    net->bwd_parts_done = 0;
    net->last_n = s.n;
    return 0;
}

int b200_backward_ft(b200_net* net, int slot, int part, int n_parts) {
    if (int rc = check_slot(net, slot, "backward_ft")) return rc;
    if (net->bwd_slot != slot) return b200::fail(B200_ERR_STATE, "backward_ft: call b200_backward_begin on slot %d first", slot);
    const bool tiled = net->bwd_tiled();
    if (n_parts < 1 || part < 0 || part >= n_parts || part != net->bwd_parts_done)
        return b200::fail(B200_ERR_ARG, "backward_ft: parts must be run in order 0..n_parts-1 (got %d of %d)", part, n_parts);
    if (n_parts > 1 && (!tiled || net->nblocks % n_parts))
        return b200::fail(B200_ERR_UNSUPPORTED, "backward_ft: %d parts need the tiled backward and must divide the %d row blocks",
                          n_parts, net->nblocks);
    if (int rc = set_device(net)) return rc;
    Slot& s = net->slots[slot];
    const b200_net_desc& d = net->d;
    cudaEvent_t* ev = net->tev[net->steps_begun % b200_net::kTimingRing];
    const int per = net->nblocks / n_parts;
    const Tensor* l0w = net->find("l0w");
    {
        b200::FtArgs fa = ft_args(net, s);
        b200::TileArgs ta = tile_args(net, s, true);
        int grid = 0;
        if (tiled) {  // this part's run of blocks
            ta.first_block = part * per;
            ta.last_block = n_parts > 1 ? (part + 1) * per : net->nblocks;
            grid = ft_backward_grid(net, s, net->sig_on);
            if (net->sig_on && (s.mma || grid != s.expect_grid))
                return b200::fail(B200_ERR_STATE, "backward_ft: the batch was uploaded before the exchange under the backward was switched on");
        }
        int rc = d.pairwise ? launch_ft_backward<true>(net, s, fa, ta, tiled, grid) : launch_ft_backward<false>(net, s, fa, ta, tiled, grid);
        if (rc) return rc;
    }
    if (part == n_parts - 1) CK(cudaEventRecord(ev[4], net->stream));
    if (d.factoriser_rows && !(net->sig_on && net->facc)) {  // (the overlapped exchange sums the reduced blocks itself)
        // sum of this part's copies of the factoriser rows; with one part: all copies, in order
        const Tensor* f = net->find("l0f");
        const int copies = (int)(l0w->n / f->n), per_part = copies / n_parts;
        if (copies % n_parts) return b200::fail(B200_ERR_UNSUPPORTED, "backward_ft: %d parts do not divide %d factoriser copies", n_parts, copies);
        b200::factoriser_grad_kernel<<<net->sm_count * 4, 256, 0, net->stream>>>(
            reinterpret_cast<const float4*>(net->G + l0w->off + (int64_t)part * per_part * f->n),
            reinterpret_cast<float4*>(net->G + f->off), (size_t)f->n / 4, per_part, part > 0);
        LAUNCHED(net);
    }
    if (part == n_parts - 1) CK(cudaEventRecord(ev[5], net->stream));
    net->bwd_parts_done = part + 1;
    net->bwd_parts = n_parts;
    return 0;
}

int b200_backward_end(b200_net* net, int slot) {
    if (int rc = check_slot(net, slot, "backward_end")) return rc;
    if (net->bwd_slot != slot || net->bwd_parts_done < 1 || net->bwd_parts_done != net->bwd_parts)
        return b200::fail(B200_ERR_STATE, "backward_end: run b200_backward_begin and every b200_backward_ft part first");
    if (int rc = set_device(net)) return rc;
    Slot& s = net->slots[slot];
    cudaEvent_t* ev = net->tev[net->steps_begun % b200_net::kTimingRing];
    CK(cudaEventRecord(ev[6], net->stream));
    // the status word travels with the step, not with the slot: once `consumed` is recorded the uploader may
    // clear and refill the slot while the update of this step is still to come
    if (net->status_slot >= 0)
        CK(cudaMemcpyAsync(net->d_status + net->updates % b200_net::kLossRing, s.dev<int>(s.off_status), sizeof(int),
                           cudaMemcpyDeviceToDevice, net->stream));
    CK(cudaEventRecord(s.consumed, net->stream));
    s.has_consumed = true;
    net->have_backward = true;
    net->step_open = true;
    net->bwd_slot = -1;
    return 0;
}

int b200_backward(b200_net* net, int slot) {
    if (int rc = b200_backward_begin(net, slot)) return rc;
    if (int rc = b200_backward_ft(net, slot, 0, 1)) return rc;
    return b200_backward_end(net, slot);
}

int b200_grad_part(b200_net* net, int part, int n_parts, int64_t* first_float, int64_t* n_floats) {
    if (!net || !first_float || !n_floats) return b200::fail(B200_ERR_ARG, "grad_part: null argument");
    const Tensor* l0w = net->find("l0w");
    if (n_parts < 1 || part < 0 || part > n_parts) return b200::fail(B200_ERR_ARG, "grad_part: part %d of %d", part, n_parts);
    if (part == n_parts) {  // the head: loss and every tensor but l0w
        *first_float = 0;
        *n_floats = l0w->off;
        return 0;
    }
    if (net->nblocks % n_parts) return b200::fail(B200_ERR_UNSUPPORTED, "grad_part: %d parts do not divide %d row blocks", n_parts, net->nblocks);
    const int64_t per = l0w->n / n_parts;
    *first_float = l0w->off + part * per;
    *n_floats = part == n_parts - 1 ? net->n_flat - *first_float : per;  // the last part takes the alignment tail
    return 0;
}

int b200_update_range(b200_net* net, float lr, float grad_factor, int64_t first_float, int64_t n_floats) {
    if (!net) return b200::fail(B200_ERR_ARG, "update_range: null net");
    if (!net->have_backward) return b200::fail(B200_ERR_STATE, "update_range: no gradients yet, call b200_backward first");
    if (first_float < 0 || n_floats < 1 || first_float + n_floats > net->n_flat || first_float % 4 || n_floats % 4)
        return b200::fail(B200_ERR_ARG, "update_range: [%lld, +%lld) is not a 4-float-aligned range of the flat buffer",
                          (long long)first_float, (long long)n_floats);
    if (int rc = set_device(net)) return rc;
    b200::AdamArgs a{};
    a.p = reinterpret_cast<float4*>(net->P);
    a.m = reinterpret_cast<float4*>(net->M);
    a.v = reinterpret_cast<float4*>(net->V);
    a.g = reinterpret_cast<const float4*>(net->G);
    a.first4 = first_float / 4;
    a.total4 = n_floats / 4;
    a.rate = lr;
    a.adj = grad_factor;
    fill_segments(net, a);
    const long long blocks = std::min<long long>((a.total4 + 255) / 256, net->sm_count * 16);
    b200::adamw_flat_kernel<<<(unsigned)blocks, 256, 0, net->stream>>>(a);
    LAUNCHED(net);
    net->weights_moved();
    return 0;
}

// ---- the data-parallel update over peer memory (one process per GPU)

int b200_exchange_export(b200_net* net, void* handles, int64_t bytes) {
    if (!net || !handles) return b200::fail(B200_ERR_ARG, "exchange_export: null argument");
    static_assert(3 * sizeof(cudaIpcMemHandle_t) == B200_EXCHANGE_HANDLE_BYTES, "handle size");
    if (bytes < B200_EXCHANGE_HANDLE_BYTES) return b200::fail(B200_ERR_ARG, "exchange_export: %d bytes are needed", B200_EXCHANGE_HANDLE_BYTES);
    if (int rc = set_device(net)) return rc;
    cudaIpcMemHandle_t h[3];
    CK(cudaIpcGetMemHandle(&h[0], net->G));
    CK(cudaIpcGetMemHandle(&h[1], net->P));
    CK(cudaIpcGetMemHandle(&h[2], net->xch_flags));
    memcpy(handles, h, sizeof h);
    return 0;
}

int b200_exchange_import(b200_net* net, int rank, int world, const void* handles, int64_t bytes) {
    if (!net || !handles) return b200::fail(B200_ERR_ARG, "exchange_import: null argument");
    if (world < 2 || world > b200::kMaxRanks || rank < 0 || rank >= world)
        return b200::fail(B200_ERR_ARG, "exchange_import: rank %d of %d (at most %d ranks)", rank, world, b200::kMaxRanks);
    if (bytes < (int64_t)world * B200_EXCHANGE_HANDLE_BYTES) return b200::fail(B200_ERR_ARG, "exchange_import: handles of %d ranks are needed", world);
    if (net->xch_world) return b200::fail(B200_ERR_STATE, "exchange_import: peers are already mapped");
    if (net->n_flat % (4 * world)) return b200::fail(B200_ERR_UNSUPPORTED, "exchange_import: the flat buffer does not split over %d ranks", world);
    if (int rc = set_device(net)) return rc;
    const cudaIpcMemHandle_t* h = static_cast<const cudaIpcMemHandle_t*>(handles);
    auto unmap_all = [&]() {
        for (int q = 0; q < world; q++)
            if (q != rank) {
                if (net->peer_g[q]) cudaIpcCloseMemHandle(net->peer_g[q]);
                if (net->peer_p[q]) cudaIpcCloseMemHandle(net->peer_p[q]);
                if (net->peer_flags[q]) cudaIpcCloseMemHandle(net->peer_flags[q]);
            }
        memset(net->peer_g, 0, sizeof net->peer_g);
        memset(net->peer_p, 0, sizeof net->peer_p);
        memset(net->peer_flags, 0, sizeof net->peer_flags);
    };
    for (int r = 0; r < world; r++) {
        if (r == rank) {
            net->peer_g[r] = net->G;
            net->peer_p[r] = net->P;
            net->peer_flags[r] = net->xch_flags;
            continue;
        }
        void* mapped[3] = {nullptr, nullptr, nullptr};
        cudaError_t e = cudaSuccess;
        for (int k = 0; k < 3 && e == cudaSuccess; k++) e = cudaIpcOpenMemHandle(&mapped[k], h[3 * r + k], cudaIpcMemLazyEnablePeerAccess);
        net->peer_g[r] = static_cast<float*>(mapped[0]);
        net->peer_p[r] = static_cast<float*>(mapped[1]);
        net->peer_flags[r] = static_cast<int*>(mapped[2]);
        if (e != cudaSuccess) {
            cudaGetLastError();
            unmap_all();
            return b200::fail(B200_ERR_CUDA, "exchange_import: cannot map the buffers of rank %d: %s", r, cudaGetErrorString(e));
        }
    }
    net->xch_rank = rank;
    net->xch_world = world;
    b200::PeerFlags f{};
    f.world = world;
    f.rank = rank;
    f.spin_limit = net->xch_spin_limit;
    for (int r = 0; r < world; r++) f.flags[r] = net->peer_flags[r];
    CK(cudaMemcpy(net->d_peers, &f, sizeof f, cudaMemcpyHostToDevice));
    return 0;
}

int b200_update_exchange_range(b200_net* net, float lr, float grad_factor, int64_t first_float, int64_t n_floats, int gather,
                               void* stream) {
    if (!net) return b200::fail(B200_ERR_ARG, "update_exchange: null net");
    if (!net->xch_world) return b200::fail(B200_ERR_STATE, "update_exchange: map the peers with b200_exchange_import first");
    if (first_float < 0 || n_floats < 1 || first_float + n_floats > net->n_flat || first_float % 4 || n_floats % 4)
        return b200::fail(B200_ERR_ARG, "update_exchange: [%lld, +%lld) is not a 4-float-aligned range of the flat buffer",
                          (long long)first_float, (long long)n_floats);
    if (int rc = set_device(net)) return rc;
    b200::ExchangeArgs x{};
    b200::AdamArgs& a = x.adam;
    a.p = reinterpret_cast<float4*>(net->P);
    a.m = reinterpret_cast<float4*>(net->M);
    a.v = reinterpret_cast<float4*>(net->V);
    a.g = nullptr;
    a.first4 = first_float / 4;
    a.total4 = n_floats / 4;
    a.rate = lr;
    a.adj = grad_factor;
    fill_segments(net, a);
    x.world = net->xch_world;
    x.store_peers = gather ? 1 : 0;
    x.head4 = kAlignFloats / 4;
    x.flags.world = net->xch_world;
    x.flags.rank = net->xch_rank;
    x.flags.spin_limit = net->xch_spin_limit;
    x.wait_ready = net->xch_wait_ready;
    for (int r = 0; r < x.world; r++) {
        x.g[r] = reinterpret_cast<const float4*>(net->peer_g[r]);
        x.p_out[r] = reinterpret_cast<float4*>(net->peer_p[r]);
        x.flags.flags[r] = net->peer_flags[r];
    }
    // On the net's own stream the kernel runs alone and takes the whole device.  On a caller's side
    // stream it runs beside the feature-transformer kernels, whose CTAs leave room for exactly one
    // such CTA per SM: more CTAs would take whole SMs away from them instead of filling the gaps.
    const long long cap = stream ? (net->exchange_ctas > 0 ? net->exchange_ctas : net->sm_count) : net->sm_count * 8;
    const long long blocks = std::min<long long>((a.total4 + 127) / 128, cap);
    cudaStream_t on = stream ? static_cast<cudaStream_t>(stream) : net->stream;
    if (net->exchange_bulk && !stream && x.store_peers) {
        // gradients fetched and weights sent by bulk copies: one CTA per SM over the tiles of this rank's share
#define BULK(W, T, S)                                                                                                           \
    do {                                                                                                                        \
        const long long tiles = (a.total4 + (T)-1) / (T);                                                                       \
        const unsigned ctas = (unsigned)std::min<long long>(net->sm_count, tiles);                                              \
        cudaFuncSetAttribute(b200::adamw_exchange_bulk_kernel<W, T, S>, cudaFuncAttributeMaxDynamicSharedMemorySize,            \
                             (int)b200::exchange_bulk_smem<W, T, S>());                                                         \
        b200::adamw_exchange_bulk_kernel<W, T, S><<<ctas, T, b200::exchange_bulk_smem<W, T, S>(), on>>>(x);                     \
    } while (0)
        const int variant = net->exchange_bulk;
        if (x.world == 2) {
            if (variant == 2) BULK(2, 512, 3);
            else if (variant == 3) BULK(2, 128, 12);
            else BULK(2, 256, 6);
        } else if (x.world == 4) {
            BULK(4, 256, 5);
        } else {
            if (variant == 2) BULK(0, 512, 1);
            else if (variant == 3) BULK(0, 128, 6);
            else BULK(0, 256, 3);
        }
#undef BULK
        LAUNCHED(net);
        net->weights_moved();
        if (first_float == 0) net->loss_in_param = true;
        return 0;
    }
    switch (x.world) {
        case 2: b200::adamw_exchange_kernel<2><<<(unsigned)blocks, 128, 0, on>>>(x); break;
        case 4: b200::adamw_exchange_kernel<4><<<(unsigned)blocks, 128, 0, on>>>(x); break;
        case 8: b200::adamw_exchange_kernel<8><<<(unsigned)blocks, 128, 0, on>>>(x); break;
        default: b200::adamw_exchange_kernel<0><<<(unsigned)blocks, 128, 0, on>>>(x); break;
    }
    LAUNCHED(net);
    net->weights_moved();
    if (first_float == 0) net->loss_in_param = true;  // the range holds the loss: it now sits in P[0]
    return 0;
}

int b200_update_exchange(b200_net* net, float lr, float grad_factor) {
    if (!net) return b200::fail(B200_ERR_ARG, "update_exchange: null net");
    if (!net->xch_world) return b200::fail(B200_ERR_STATE, "update_exchange: map the peers with b200_exchange_import first");
    if (!net->have_backward) return b200::fail(B200_ERR_STATE, "update_exchange: no gradients yet, call b200_backward first");
    const int64_t per = net->n_flat / net->xch_world;
    if (int rc = set_device(net)) return rc;
    // fences without a collective: tell the peers that this rank's gradients are complete; the exchange
    // kernel waits for every peer's word before it reads; afterwards the same once more for "finished",
    // so that nobody overwrites gradients or reads weights while a peer's kernel is still at work
    b200::PeerFlags f{};
    f.world = net->xch_world;
    f.rank = net->xch_rank;
    f.spin_limit = net->xch_spin_limit;
    for (int r = 0; r < f.world; r++) f.flags[r] = net->peer_flags[r];
    const int step = ++net->xch_step;
    b200::peer_signal_kernel<<<1, 32, 0, net->stream>>>(f, b200::kFlagReady, step);
    LAUNCHED(net);
    net->xch_wait_ready = step;
    int rc = b200_update_exchange_range(net, lr, grad_factor, net->xch_rank * per, per, 1, nullptr);
    net->xch_wait_ready = 0;
    if (rc) return rc;
    b200::peer_signal_kernel<<<1, 32, 0, net->stream>>>(f, b200::kFlagDone, step);
    LAUNCHED(net);
    b200::peer_wait_kernel<<<1, 32, 0, net->stream>>>(f, b200::kFlagDone, step);
    LAUNCHED(net);
    net->loss_in_param = true;  // rank 0's share starts with the loss and stores it to every rank
    net->xch_fenced_used = true;
    return 0;
}

// One data-parallel step with the exchange under the backward pass (see adamw_exchange_overlap_kernel).
int b200_step_exchange(b200_net* net, int slot, float lr, float grad_factor) {
    if (!net) return b200::fail(B200_ERR_ARG, "step_exchange: null net");
    if (!net->xch_world) return b200::fail(B200_ERR_STATE, "step_exchange: map the peers with b200_exchange_import first");
    const b200_net_desc& d = net->d;
    const Tensor* l0w = net->find("l0w");
    const Tensor* l0f = d.factoriser_rows ? net->find("l0f") : nullptr;
    const int64_t block_floats = (int64_t)d.ft_block_rows * d.ft_out;
    if (!net->bwd_tiled() || !net->tiled_promised || net->nblocks > b200::kMaxSignalBlocks)
        return b200::fail(B200_ERR_UNSUPPORTED, "step_exchange: needs the tiled backward (ft_block_rows > 0) and at most %d row blocks",
                          b200::kMaxSignalBlocks);
    if (block_floats % (4 * net->xch_world)) return b200::fail(B200_ERR_UNSUPPORTED, "step_exchange: a row block does not split over %d ranks", net->xch_world);
    if (l0f && !net->facc) return b200::fail(B200_ERR_UNSUPPORTED, "step_exchange: the factoriser must have as many rows as a row block");
    if (int rc = b200_backward_begin(net, slot)) return rc;
    Slot& s = net->slots[slot];
    const int step = ++net->xch_step;

    b200::OverlapArgs o{};
    b200::ExchangeArgs& x = o.x;
    b200::AdamArgs& a = x.adam;
    a.p = reinterpret_cast<float4*>(net->P);
    a.m = reinterpret_cast<float4*>(net->M);
    a.v = reinterpret_cast<float4*>(net->V);
    a.rate = lr;
    a.adj = grad_factor;
    fill_segments(net, a);
    o.l0f_seg = -1;
    for (int i = 0; i < a.nseg; i++) {
        if (&net->tensors[i] == l0w) o.l0w_seg = i;
        if (&net->tensors[i] == l0f) o.l0f_seg = i;
    }
    x.world = net->xch_world;
    x.store_peers = 1;
    x.head4 = kAlignFloats / 4;
    x.flags.world = net->xch_world;
    x.flags.rank = net->xch_rank;
    x.flags.spin_limit = net->xch_spin_limit;
    for (int r = 0; r < x.world; r++) {
        x.g[r] = reinterpret_cast<const float4*>(net->peer_g[r]);
        x.p_out[r] = reinterpret_cast<float4*>(net->peer_p[r]);
        x.flags.flags[r] = net->peer_flags[r];
    }
    o.step = step;
    o.nblocks = net->nblocks;
    o.l0w4 = l0w->off / 4;
    o.block4 = block_floats / 4;
    o.l0f4 = l0f ? l0f->off / 4 : 0;
    o.facc = l0f ? reinterpret_cast<float4*>(net->facc) : nullptr;

    // the exchange kernel goes first, on its own stream: it is resident (or first in line for an SM) by the
    // time the backward's CTAs arrive, and it depends on them, never they on it
    CK(cudaEventRecord(net->xch_fork, net->stream));
    CK(cudaStreamWaitEvent(net->xch_stream, net->xch_fork, 0));
    const int ctas = std::min(net->overlap_ctas, net->sm_count - 1);
    switch (x.world) {
        case 2: b200::adamw_exchange_overlap_kernel<2><<<ctas, b200::kOverlapThreads, b200::kOverlapSmem, net->xch_stream>>>(o); break;
        case 4: b200::adamw_exchange_overlap_kernel<4><<<ctas, b200::kOverlapThreads, b200::kOverlapSmem, net->xch_stream>>>(o); break;
        case 8: b200::adamw_exchange_overlap_kernel<8><<<ctas, b200::kOverlapThreads, b200::kOverlapSmem, net->xch_stream>>>(o); break;
        default: b200::adamw_exchange_overlap_kernel<0><<<ctas, b200::kOverlapThreads, b200::kOverlapSmem, net->xch_stream>>>(o); break;
    }
    LAUNCHED(net);
    b200::PeerFlags f = x.flags;
    // ... and behind it the closing fence: every rank's kernel has finished before anyone reuses gradients or weights
    b200::peer_signal_kernel<<<1, 32, 0, net->xch_stream>>>(f, b200::kFlagDone, step);
    LAUNCHED(net);
    b200::peer_wait_kernel<<<1, 32, 0, net->xch_stream>>>(f, b200::kFlagDone, step);
    LAUNCHED(net);
    CK(cudaEventRecord(net->xch_join, net->xch_stream));

    // the backward, announcing its row blocks as they finish
    net->sig_on = true;
    net->sig_value = step;
    {
        b200::TileArgs ta = tile_args(net, s, true);
        b200::bucket_presignal_kernel<<<1, 256, 0, net->stream>>>(ta.sig, net->nblocks);
        LAUNCHED(net);
    }
    int rc = b200_backward_ft(net, slot, 0, 1);
    net->sig_on = false;
    if (rc) return rc;
    b200::peer_signal_kernel<<<1, 32, 0, net->stream>>>(f, b200::kFlagReady, step);  // bias and dense gradients too
    LAUNCHED(net);
    if (int rc2 = b200_backward_end(net, slot)) return rc2;
    CK(cudaStreamWaitEvent(net->stream, net->xch_join, 0));
    net->loss_in_param = true;  // every rank reduced the loss into float 0 of its parameter buffer
    net->xch_fenced_used = true;
    net->weights_moved();
    return b200_update_end(net);
}

int b200_grad_zero_range(b200_net* net, int64_t first_float, int64_t n_floats) {
    if (!net) return b200::fail(B200_ERR_ARG, "grad_zero_range: null net");
    if (first_float < 0 || n_floats < 1 || first_float + n_floats > net->n_flat)
        return b200::fail(B200_ERR_ARG, "grad_zero_range: [%lld, +%lld) is outside the flat buffer", (long long)first_float, (long long)n_floats);
    if (int rc = set_device(net)) return rc;
    CK(cudaMemsetAsync(net->G + first_float, 0, (size_t)n_floats * 4, net->stream));
    return 0;
}

// Ranger: every k-th step the fast weights are pulled towards the slow ones, which then follow.  Due after the update that is
// about to be counted?
static bool lookahead_due(const b200_net* net) {
    for (const Tensor& t : net->tensors)
        if (net->S && t.opt_kind == B200_OPT_RANGER && (net->opt_step + 1) % t.lookahead_k == 0) return true;
    return false;
}
static int launch_lookahead(b200_net* net) {  // (after the count)
    b200::LookaheadArgs la{};
    la.p = reinterpret_cast<float4*>(net->P);
    la.slow = reinterpret_cast<float4*>(net->S);
    la.total4 = net->n_flat / 4;
    la.nseg = (int)net->tensors.size();
    for (int i = 0; i < la.nseg; i++) {
        const Tensor& t = net->tensors[i];
        la.begin4[i] = t.off / 4;
        la.end4[i] = (t.off + t.n + 3) / 4;
        const bool due = t.opt_kind == B200_OPT_RANGER && net->opt_step % t.lookahead_k == 0;
        la.alpha[i] = due ? t.alpha : -1.f;
        la.one_minus[i] = 1.0f - t.alpha;
    }
    b200::lookahead_kernel<<<net->sm_count * 8, 256, 0, net->stream>>>(la);
    LAUNCHED(net);
    net->weights_moved();
    return 0;
}

int b200_update_end(b200_net* net) {
    if (!net) return b200::fail(B200_ERR_ARG, "update_end: null net");
    if (!net->have_backward) return b200::fail(B200_ERR_STATE, "update_end: no gradients yet");
    if (int rc = set_device(net)) return rc;
    const int ring = (int)(net->updates % b200_net::kLossRing);
    CK(cudaMemcpyAsync(net->h_loss + ring, net->loss_in_param ? net->P : net->G, sizeof(float), cudaMemcpyDeviceToHost, net->stream));
    net->loss_in_param = false;
    if (net->status_slot >= 0) {
        CK(cudaMemcpyAsync(net->h_status + ring, net->d_status + ring, sizeof(int), cudaMemcpyDeviceToHost, net->stream));
    } else {
        net->h_status[ring] = 0;
    }
    if (net->xch_fenced_used) {
        // report the word with this step, then clear it: a later good step starts clean
        CK(cudaMemcpyAsync(net->h_xstatus + 4 * ring, net->xch_flags + b200::kFlagTimeout, 4 * sizeof(int), cudaMemcpyDeviceToHost, net->stream));
        CK(cudaMemsetAsync(net->xch_flags + b200::kFlagTimeout, 0, 4 * sizeof(int), net->stream));
    }
    CK(cudaEventRecord(net->loss_ev[ring], net->stream));
    net->updates++;
    const bool lookahead = lookahead_due(net);
    net->opt_step++;
    if (lookahead)
        if (int rc = launch_lookahead(net)) return rc;
    if (int rc = refresh_table(net, net->last_n)) return rc;
    if (net->step_open) {  // close the timed step begun by the matching backward
        CK(cudaEventRecord(net->tev[net->steps_begun % b200_net::kTimingRing][7], net->stream));
        net->steps_begun++;
        net->steps_done = net->steps_begun;
        net->step_open = false;
    }
    return 0;
}

int b200_update(b200_net* net, float lr, float grad_factor) {
    if (!net) return b200::fail(B200_ERR_ARG, "update: null net");
    if (int rc = b200_update_range(net, lr, grad_factor, 0, net->n_flat)) return rc;
    return b200_update_end(net);
}

// A whole step enqueued at once: nothing is observed between its phases, so its kernels are chained (launch.cuh), keep their
// own time, and the update forms the factoriser's gradient, the first dense layer's tables and the read-back itself.
static int step_chained(b200_net* net, Slot& s, int slot, float lr, float grad_factor) {
    const b200_net_desc& d = net->d;
    CK(cudaStreamWaitEvent(net->stream, s.ready, 0));
    net->trains = true;
    if (int rc = refresh_table(net, s.n)) return rc;
    const int ring = (int)(net->updates % b200_net::kLossRing);
    // a small gradient buffer is cleared by the forward kernel; a large one would hold it up
    const bool clear_here = net->n_flat <= kClearInForward;
    if (!clear_here)
        if (int rc = clear_gradients_aside(net)) return rc;
    if (int rc = forward_prepare(net, s, true)) return rc;
    const bool bwd_tiled = net->bwd_tiled();
    if (bwd_tiled && !s.csr_built)
        if (int rc = build_csr(net, s, net->stream)) return rc;
    {
        const bool tiled = net->fwd_tiled(s.n);
        b200::FtArgs fa = ft_args(net, s);
        b200::TileArgs ta = tile_args(net, s, false);
        fa.stamp = net->stamp(0);
        fa.stamp_end = net->stamp(7);
        if (clear_here) {
            fa.zero = reinterpret_cast<float4*>(net->G);
            fa.zero4 = net->n_flat / 4;
        }
        const int grid = tiled ? ft_forward_grid(net, s) : 0;
        int rc = d.pairwise ? launch_ft_forward<true>(net, fa, ta, tiled, grid) : launch_ft_forward<false>(net, fa, ta, tiled, grid);
        if (rc) return rc;
    }
    if (int rc = forward_dense(net, s, true)) return rc;
    if (!net->dense_one()) {
        b200::DenseArgs da = dense_args(net, s, true);
        da.stamp = net->stamp(2);
        DISPATCH_M(d.dense_out[0], launch_dense_dx<MM>(net, da, s.n_dtiles));
        LAUNCHED(net);
        if (int rc = launch_dense_grads(net, s)) return rc;
    }
    {
        b200::FtArgs fa = ft_args(net, s);
        b200::TileArgs ta = tile_args(net, s, true);
        fa.stamp = net->stamp(3);
        const int grid = bwd_tiled ? ft_backward_grid(net, s, false) : 0;
        int rc = d.pairwise ? launch_ft_backward<true>(net, s, fa, ta, bwd_tiled, grid) : launch_ft_backward<false>(net, s, fa, ta, bwd_tiled, grid);
        if (rc) return rc;
    }
    const bool lookahead = lookahead_due(net);
    {
        b200::StepUpdateArgs u{};
        b200::AdamArgs& a = u.adam;
        a.p = reinterpret_cast<float4*>(net->P);
        a.m = reinterpret_cast<float4*>(net->M);
        a.v = reinterpret_cast<float4*>(net->V);
        a.rate = lr;
        a.adj = grad_factor;
        fill_segments(net, a);
        u.g = reinterpret_cast<float4*>(net->G);
        const Tensor *l0w = net->find("l0w"), *l0f = d.factoriser_rows ? net->find("l0f") : nullptr, *l1w = net->find("l1w");
        u.l0f_seg = u.l0w_seg = -1;
        if (l0f)
            for (int i = 0; i < a.nseg; i++) {
                if (&net->tensors[i] == l0w) u.l0w_seg = i;
                if (&net->tensors[i] == l0f) u.l0f_seg = i;
            }
        u.rest4 = l0f ? l0w->off / 4 : net->n_flat / 4;
        u.l0w4 = l0w->off / 4;
        u.l0f4 = l0f ? l0f->off / 4 : 0;
        u.block4 = l0f ? l0f->n / 4 : 0;
        u.copies = l0f ? (int)(l0w->n / l0f->n) : 0;
        u.l1w4_begin = l1w->off / 4;
        u.l1w4_end = lookahead ? u.l1w4_begin : (l1w->off + l1w->n + 3) / 4;  // (the lookahead moves the weights once more)
        u.K1 = net->D1();
        u.O = d.n_out_buckets;
        u.M1 = d.dense_out[0];
        if (!lookahead && !net->dense_mma()) net->w1_now ^= 1;
        u.w1g = net->w1g_now();
        u.w1f = net->w1f;
        u.w1d = net->w1d;
        u.loss = net->G;
        u.status = net->status_slot >= 0 ? s.dev<int>(s.off_status) : nullptr;
        u.h_loss = net->h_loss + ring;
        u.h_status = net->h_status + ring;
        u.stamps = net->stamp(0);
        net->update_copies = l0f && !b200::update_by_thread(u.copies, u.block4, net->sm_count);
        if (net->update_copies) {
            const b200::CopiesShape shape = b200::copies_shape(u.copies);
            const int threads = shape.threads(), wide = 32 * shape.sets;
            const int rest = (int)((u.rest4 - u.block4 + threads - 1) / threads), tiles = (int)((u.block4 + wide - 1) / wide);
            CK(b200::launch_step(true, shape.copies == b200::kUpdWarps ? b200::step_update_copies_kernel<true> : b200::step_update_copies_kernel<false>, rest + tiles, threads, 0, net->stream, u, rest, shape));
        } else {
            const long long items = std::max(u.rest4, u.block4);
            CK(b200::launch_step(true, b200::step_update_kernel, (unsigned)std::min<long long>((items + 255) / 256, net->sm_count * 32), 256, 0, net->stream, u));
        }
        LAUNCHED(net);
        net->weights_moved();
        net->w1_dirty = lookahead;
    }
    CK(cudaEventRecord(s.consumed, net->stream));
    s.has_consumed = true;
    CK(cudaEventRecord(net->loss_ev[ring], net->stream));
    net->last_n = s.n;
    net->have_backward = true;
    net->loss_in_param = false;
    net->updates++;
    net->opt_step++;
    net->stamped[net->steps_begun % b200_net::kTimingRing] = true;
    net->steps_begun++;
    net->steps_done = net->steps_begun;
    if (lookahead) {
        if (int rc = launch_lookahead(net)) return rc;
        if (int rc = refresh_table(net, net->last_n)) return rc;
    }
    return 0;
}

int b200_step(b200_net* net, int slot, float lr, float grad_factor) {
    if (int rc = check_slot(net, slot, "step")) return rc;
    if (net->fwd_slot < 0 && net->bwd_slot < 0 && !net->manual_grad_zero && !net->sig_on && !net->xch_fenced_used) {
        if (int rc = set_device(net)) return rc;
        net->chained = true;
        const int rc = step_chained(net, net->slots[slot], slot, lr, grad_factor);
        net->chained = false;
        return rc;
    }
    if (int rc = b200_backward(net, slot)) return rc;
    return b200_update(net, lr, grad_factor);
}

int b200_grad_buffer(b200_net* net, void** device_ptr, int64_t* n_floats) {
    if (!net || !device_ptr || !n_floats) return b200::fail(B200_ERR_ARG, "grad_buffer: null argument");
    *device_ptr = net->G;
    *n_floats = net->n_flat;
    return 0;
}

int b200_flat_buffer(b200_net* net, int kind, void** device_ptr, int64_t* n_floats) {
    if (!net || !device_ptr || !n_floats) return b200::fail(B200_ERR_ARG, "flat_buffer: null argument");
    float* base = kind_base(net, kind);
    if (!base) return b200::fail(B200_ERR_ARG, "flat_buffer: unknown kind %d", kind);
    *device_ptr = base;
    *n_floats = net->n_flat;
    return 0;
}

static int check_waits(b200_net* net) {
    if (!*(volatile int*)net->h_gave_up) return 0;
    *net->h_gave_up = 0;
    return b200::fail(B200_ERR_CUDA, "a kernel gave up waiting for its own copies; the results of that pass are not valid");
}

int b200_loss_of(b200_net* net, int steps_back, float* loss_sum) {
    if (!net || !loss_sum) return b200::fail(B200_ERR_ARG, "loss: null argument");
    if (steps_back < 0 || steps_back >= b200_net::kLossRing - 1)
        return b200::fail(B200_ERR_ARG, "loss: only the last %d updates are kept", b200_net::kLossRing - 1);
    if (net->updates <= steps_back) return b200::fail(B200_ERR_STATE, "loss: that update has not run yet");
    if (int rc = set_device(net)) return rc;
    const int ring = (int)((net->updates - 1 - steps_back) % b200_net::kLossRing);
    CK(cudaEventSynchronize(net->loss_ev[ring]));
    *loss_sum = net->h_loss[ring];
    if (int rc = check_waits(net)) return rc;
    if (net->h_xstatus[4 * ring]) {
        const int* x = net->h_xstatus + 4 * ring;
        const int base = x[1], value = x[2], who = x[3];
        net->h_xstatus[4 * ring] = 0;
        if (value == 0)
            return b200::fail(B200_ERR_STATE, "data-parallel exchange: a peer did not reach the fence in time (reported by another rank); "
                                              "the update of this step is not valid");
        return b200::fail(B200_ERR_STATE,
                          "data-parallel exchange: a peer did not reach the fence in time (rank %d never announced %s%d of step %d); the "
                          "update of this step is not valid",
                          who, base >= b200::kFlagBucket ? "row block " : base >= b200::kFlagDone ? "the end of its exchange, fence " : "its gradients, fence ",
                          base >= b200::kFlagBucket ? (base - b200::kFlagBucket) / b200::kMaxRanks : base, value);
    }
    if (net->h_status[ring] & b200::kStatusOutsideBlock) {
        net->h_status[ring] = 0;
        return b200::fail(B200_ERR_DATA,
                          "a feature index fell outside the row block of its position (ft_block_rows=%d): those "
                          "features were ignored; create the network with ft_block_rows=0 for such inputs",
                          net->d.ft_block_rows);
    }
    return 0;
}

int b200_loss(b200_net* net, float* loss_sum) { return b200_loss_of(net, 0, loss_sum); }

int b200_forward(b200_net* net, int slot, float* out_host) {
    if (int rc = check_slot(net, slot, "forward")) return rc;
    if (!out_host) return b200::fail(B200_ERR_ARG, "forward: null output");
    if (int rc = set_device(net)) return rc;
    Slot& s = net->slots[slot];
    CK(cudaStreamWaitEvent(net->stream, s.ready, 0));
    if (int rc = refresh_table(net, s.n)) return rc;
    // nothing is observed between the kernels of an evaluation either; the outputs leave by a kernel, because a copy behind one
    // starts 10 us late
    net->chained = true;
    int rc = forward_part(net, s, false);
    if (!rc && s.n > kDirectOutputs) {
        const int ctas = std::min(net->sm_count, (s.n + 255) / 256);
        if (b200::launch_step(true, b200::copy_outputs_kernel, ctas, 256, 0, net->stream, net->out, net->h_out, s.n) != cudaSuccess)
            rc = b200::fail(B200_ERR_CUDA, "forward: launching the output copy failed: %s", cudaGetErrorString(cudaGetLastError()));
        net->launches++;
    }
    net->chained = false;
    if (rc) return rc;
    CK(cudaEventRecord(s.consumed, net->stream));
    s.has_consumed = true;
    net->last_n = s.n;
    CK(cudaStreamSynchronize(net->stream));
    memcpy(out_host, net->h_out, (size_t)s.n * sizeof(float));
    if (int rc = check_waits(net)) return rc;
    return 0;
}

int b200_sync(b200_net* net) {
    if (!net) return b200::fail(B200_ERR_ARG, "sync: null net");
    if (int rc = set_device(net)) return rc;
    CK(cudaStreamSynchronize(net->copy_stream));
    CK(cudaStreamSynchronize(net->stream));
    return 0;
}

int b200_get_timings(b200_net* net, b200_timings* out) {
    if (!net || !out) return b200::fail(B200_ERR_ARG, "get_timings: null argument");
    if (int rc = set_device(net)) return rc;
    memset(out, 0, sizeof *out);
    const int64_t first = std::max(net->timing_origin, net->steps_done - b200_net::kTimingRing);
    const int64_t count = net->steps_done - first;
    net->timing_origin = net->steps_done;
    if (count < 1) return b200::fail(B200_ERR_STATE, "get_timings: no complete step since the last call");
    CK(cudaStreamSynchronize(net->stream));
    // events: 0 start, 1 FT forward, 2 dense forward, 3 dx, 4 FT backward, 5 factoriser sums,
    // 6 dense weight gradients, 7 update
    double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    std::vector<unsigned long long> stamps((size_t)b200_net::kTimingRing * b200_net::kTimingEvents);
    CK(cudaMemcpy(stamps.data(), net->d_stamps, stamps.size() * sizeof(stamps[0]), cudaMemcpyDeviceToHost));
    for (int64_t i = first; i < net->steps_done; i++) {
        if (net->stamped[i % b200_net::kTimingRing]) {
            // whole steps: starts of FT forward, dense forward, dx, FT backward and update, end of the update
            unsigned long long* t = stamps.data() + (i % b200_net::kTimingRing) * b200_net::kTimingEvents;
            if (net->dense_one()) t[2] = t[3];
            const int from[7] = {0, 1, 2, 3, 4, 4, 4}, to[7] = {1, 2, 3, 4, 4, 4, 7};
            for (int k = 0; k < 7; k++) acc[k] += (double)(int64_t)(t[to[k]] - t[from[k]]) * 1e-6;
            acc[7] += (double)(int64_t)(t[7] - t[0]) * 1e-6;
            continue;
        }
        cudaEvent_t* ev = net->tev[i % b200_net::kTimingRing];
        float ms = 0.f;
        for (int k = 0; k < 7; k++) {
            CK(cudaEventElapsedTime(&ms, ev[k], ev[k + 1]));
            acc[k] += ms;
        }
        CK(cudaEventElapsedTime(&ms, ev[0], ev[7]));
        acc[7] += ms;
    }
    const double inv = 1.0 / (double)count;
    out->ft_forward = (float)(acc[0] * inv);
    out->dense_forward = (float)(acc[1] * inv);
    out->dense_backward = (float)((acc[2] + acc[5]) * inv);
    out->ft_backward = (float)(acc[3] * inv);
    out->factoriser_grad = (float)(acc[4] * inv);
    out->optimiser = (float)(acc[6] * inv);
    out->total = (float)(acc[7] * inv);
    out->steps = (int32_t)count;
    return 0;
}

int b200_net_get_stat(b200_net* net, const char* key, int64_t* value) {
    if (!net || !key || !value) return b200::fail(B200_ERR_ARG, "get_stat: null argument");
    if (!strcmp(key, "launches")) *value = net->launches;
    else if (!strcmp(key, "h2d_bytes")) *value = net->h2d_bytes;
    else if (!strcmp(key, "flat_floats")) *value = net->n_flat;
    else if (!strcmp(key, "ft_tiled")) *value = (net->fwd_tiled() ? 1 : 0) + (net->bwd_tiled() ? 2 : 0);
    else if (!strcmp(key, "ft_forward")) *value = net->fwd_last;
    else if (!strcmp(key, "ft_products")) *value = net->products_last ? 1 : 0;
    else if (!strcmp(key, "ft_chunk")) *value = net->chunk_last;
    else if (!strcmp(key, "update_copies")) *value = net->update_copies ? 1 : 0;
    else if (!strcmp(key, "slow_weights")) *value = net->S ? 1 : 0;
    else if (!strcmp(key, "optimiser_steps")) *value = net->opt_step;
    else return b200::fail(B200_ERR_ARG, "get_stat: unknown key '%s'", key);
    return 0;
}

int b200_net_get_activation(b200_net* net, int which, float* host, int64_t n) {
    if (!net || !host) return b200::fail(B200_ERR_ARG, "get_activation: null argument");
    const int64_t B = net->last_n;
    const float* src = nullptr;
    int64_t want = 0;
    switch (which) {
        case 0: src = net->x; want = B * net->D1(); break;
        case 1: src = net->u; want = net->d.pairwise ? B * 2 * net->d.ft_out : 0; break;
        case 2: src = net->dx; want = B * net->D1(); break;
        case 3: src = net->out; want = B; break;
        default: return b200::fail(B200_ERR_ARG, "get_activation: unknown buffer %d", which);
    }
    if (!src || want == 0) return b200::fail(B200_ERR_STATE, "get_activation: buffer %d is not used by this network", which);
    if (n != want) return b200::fail(B200_ERR_ARG, "get_activation: buffer %d holds %lld values, %lld asked", which, (long long)want, (long long)n);
    if (int rc = set_device(net)) return rc;
    if (which == 2 && net->dense_one()) {
        if (int rc = form_dx(net)) return rc;
        // the last pass may have been an evaluation of more positions: those have no gradient
        if (B > net->grad_n) CK(cudaMemsetAsync(net->dx + net->grad_n * (int64_t)net->D1(), 0, (size_t)(B - net->grad_n) * net->D1() * sizeof(float), net->stream));
    }
    CK(cudaStreamSynchronize(net->stream));
    CK(cudaMemcpy(host, src, n * sizeof(float), cudaMemcpyDeviceToHost));
    if (which == 0 && net->keep_root())
        for (int64_t i = 0; i < n; i++) host[i] *= host[i];
    return 0;
}

}  // extern "C"
