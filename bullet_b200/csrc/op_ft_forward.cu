// Operator-level entry points: the feature-transformer forward on caller-owned device memory.
//
// b200_op_ft_forward computes, for both perspectives of n positions, what the reference's
// graph computes with SparseMatmul::evaluate (crates/compiler/src/tensor/operation/linear/sparse.rs:86-119)
// followed by the bias add (crates/compiler/src/model/builder.rs:145-147), the activation
// (crates/compiler/src/tensor/operation/autograd/dfo.rs:47-88), the optional pairwise product
// (model/builder.rs:390-393) and the stm|nstm concat (model/builder.rs:375-388) — the same
// kernel b200_step runs, but without a b200_net: table, bias, packed index lists and outputs are
// device pointers of the caller.
//
// The tiled kernel visits (position, perspective) pairs grouped by the table row block their
// features live in; the grouping (kernels_group.cuh) is built on the device into scratch memory.
// b200_op_ft_forward takes that scratch from a memory pool of its own; b200_op_ft_forward_noalloc keeps
// it in a fixed array that is part of the library image.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <mutex>

#include "../../include/bullet_b200.h"
#include "common.h"
#include "kernels_group.cuh"
#include "op_pool.h"

#define CK(call)                                                                                          \
    do {                                                                                                  \
        cudaError_t e_ = (call);                                                                          \
        if (e_ != cudaSuccess)                                                                            \
            return b200::fail(B200_ERR_CUDA, "%s failed: %s (%d) at %s:%d", #call, cudaGetErrorString(e_), \
                              (int)e_, __FILE__, __LINE__);                                               \
    } while (0)

namespace {

constexpr int kMaxBlocks = 1024;  // table row blocks the grouping supports

// Scratch layout, in ints, every section on a 256-byte boundary: the blocks' first pairs and a status word, per pair its
// block and list length [2n], (pair id, rows) [2n] and the prepared row lists [2n][nnz rounded up to 8] as u16, then the
// histograms of the grouping's first pass, or its counters where there are more blocks than its windows hold.
constexpr size_t kSectionAlign = 64;  // ints
constexpr size_t align_ints(size_t v) { return (v + kSectionAlign - 1) / kSectionAlign * kSectionAlign; }
constexpr size_t kStatusAt = kMaxBlocks + 1;
constexpr size_t kScratchHeader = align_ints(kMaxBlocks + 2);
constexpr int list_len(int nnz) { return (nnz + 7) & ~7; }  // 16-byte groups of u16 row indices
constexpr size_t hist_ints(int n, int nblocks) {
    return nblocks > b200::kGroupMaxBlocks ? align_ints(3 * (size_t)(nblocks + 3))
                                           : align_ints((size_t)((n + b200::kGroupPositions - 1) / b200::kGroupPositions + 1) * (nblocks + 1));
}
constexpr size_t scratch_ints(int n, int nnz, int nblocks) {
    return kScratchHeader + align_ints((size_t)2 * n) + align_ints((size_t)4 * n) + (size_t)n * list_len(nnz) + hist_ints(n, nblocks);
}

// Scratch of b200_op_ft_forward_noalloc: room for B200_OP_NOALLOC_MAX_POSITIONS positions of
// up to 32 index slots (about 2.7 MB).  It is a file-scope device array, so every GPU on
// which the library is loaded carries it from load until the process exits, and every call
// on that GPU uses the same bytes.
constexpr size_t kStaticInts = scratch_ints(B200_OP_NOALLOC_MAX_POSITIONS, 32, b200::kGroupMaxBlocks);
static __device__ __align__(256) int g_op_scratch[kStaticInts];

// A call's status word: memory of the library image that both sides may touch at any time, and that the kernels touch only if
// there is something to report, so that nothing has to be allocated and nothing copied back.  (A 4-byte copy behind the forward
// takes 10 us: b200_op_ft_forward_noalloc on 2048 positions, king buckets, width 1024: 72 us with it, 62 without.)  A call holds a
// word from its first kernel until its stream has finished.  A call that finds none free, or a device that cannot share such
// memory while it is running, has the word in its scratch and copies it back.
constexpr int kStatusWords = 64, kStatusStride = 16;  // (a cache line each)
static __managed__ int g_op_status[kStatusWords * kStatusStride];

// Whether `device` can share g_op_status; asks the runtime once per device, and has the words stay in host memory.
bool shares_status(int device) {
    constexpr int kDevices = 64;
    static std::atomic<signed char> known[kDevices];  // 0 not asked yet, 1 yes, -1 no
    if (device < 0 || device >= kDevices) return false;
    if (const signed char k = known[device]) return k > 0;
    int concurrent = 0;
    if (cudaDeviceGetAttribute(&concurrent, cudaDevAttrConcurrentManagedAccess, device) != cudaSuccess) concurrent = 0;
    if (concurrent) {  // (hints: without them a report would move the page to the device and back)
        cudaMemAdvise(g_op_status, sizeof g_op_status, cudaMemAdviseSetPreferredLocation, cudaCpuDeviceId);
        cudaMemAdvise(g_op_status, sizeof g_op_status, cudaMemAdviseSetAccessedBy, device);
    }
    cudaGetLastError();
    known[device] = concurrent ? 1 : -1;
    return concurrent != 0;
}

struct StatusWord {
    StatusWord(int device, cudaStream_t on) : stream(on) {
        if (!shares_status(device)) return;
        for (int k = 0; k < kStatusWords && !status; k++) {
            bool free = false;
            if (taken()[k].compare_exchange_strong(free, true)) at = k, status = g_op_status + kStatusStride * k;
        }
        if (status) *status = 0;
    }
    ~StatusWord() {
        if (!status) return;
        if (!finished) cudaStreamSynchronize(stream);  // a call that failed half way: kernels may still be about to write
        taken()[at] = false;
    }
    StatusWord(const StatusWord&) = delete;
    StatusWord& operator=(const StatusWord&) = delete;
    static std::atomic<bool>* taken() {
        static std::atomic<bool> flags[kStatusWords];
        return flags;
    }
    cudaStream_t stream;
    int* status = nullptr;
    int at = 0;
    bool finished = false;
};

int check_op(const b200_ft_op* op, const char* who) {
    if (!op) return b200::fail(B200_ERR_ARG, "%s: null operator description", who);
    if (!op->table || !op->bias || !op->idx_stm || !op->idx_nstm || !op->x || (op->pairwise && !op->u))
        return b200::fail(B200_ERR_ARG, "%s: null device pointer", who);
    if (op->n < 1) return b200::fail(B200_ERR_ARG, "%s: n must be positive", who);
    if (op->n > INT32_MAX / 4) return b200::fail(B200_ERR_ARG, "%s: at most %d positions per call", who, INT32_MAX / 4);
    if (op->nnz < 1 || op->nnz > 64 || op->n_inputs < 1 || op->n_inputs > 65534)
        return b200::fail(B200_ERR_UNSUPPORTED, "%s: nnz must be in [1, 64] and n_inputs in [1, 65534]", who);
    if (op->ft_act != B200_ACT_CRELU && op->ft_act != B200_ACT_SCRELU)
        return b200::fail(B200_ERR_UNSUPPORTED, "%s: activation must be CReLU or SCReLU", who);
    if (op->pairwise && op->ft_act != B200_ACT_CRELU) return b200::fail(B200_ERR_UNSUPPORTED, "%s: pairwise needs CReLU", who);
    const int R = op->ft_block_rows;
    if (R < 1 || op->n_inputs % R || op->ft_out < 64 || op->ft_out % b200::kTileCols || op->n_inputs / R > kMaxBlocks ||
        !b200::ft_fwd_fits(R, list_len(op->nnz)))
        return b200::fail(B200_ERR_UNSUPPORTED,
                          "%s: needs ft_block_rows > 0 dividing n_inputs (at most about 800 rows, at most %d blocks) "
                          "and ft_out a multiple of 64",
                          who, kMaxBlocks);
    return 0;
}

// Few positions are not worth grouping, nor the table's way through shared memory: the gather forward (one kernel, rows from L2)
// takes them as they are.  Its time goes with the bytes of the rows, which the slots bound, the tiled form's
// with the tiles besides, of which a CTA has at least one.  Whole call on a B200, us, gathered / grouped, by MB of slots (half of them active; all):
//   512 tiles and more: 16 blocks of 768 rows x 2048 columns pairwise 1500 77 / 93; 107 / 111; 40 blocks x 2048 1500 91 / 133; 121 / 154; 96 rows x 64 blocks x 512 1500 71 / 115; 101 / 130
//   a tile for every SM: 16 blocks of 768 rows x 1024 890 45 / 57; 66 / 67, 1150 54 / 64; 77 / 78, 1500 65 / 72; 99 / 93; pairwise 1500 73 / 80; 105 / 100
//   16 tiles and more: eight blocks of 768 rows x 1024 700 40 / 46; 56 / 55, 1000 49 / 52; 71 / 65; four x 512 890 44 / 49; 63 / 61, 1000 48 / 51; 69 / 64
//   147 rows x 1024 890 37 / 60; 49 / 70, 1000 42 / 64; 60 / 75
//   fewer, which most SMs then share: 147 rows x 256 570 29 / 38; 36 / 50; 768 rows x 128 570 39 / 45; 49 / 54, 700 -, 46; -, 52
// The lines lie where full lists meet.  Outputs that start on any float are for the tiled kernel.
constexpr long long kGatherMostManyTiles = 1536LL << 20, kGatherMost = 1152LL << 20, kGatherMostFewTiles = 896LL << 20, kGatherMostFewestTiles = 576LL << 20;
bool few_positions(const b200_ft_op* op, int sms) {
    if (((uintptr_t)op->bias | (uintptr_t)op->x | (op->pairwise ? (uintptr_t)op->u : 0)) & 15) return false;
    const long long tiles = (long long)(op->n_inputs / op->ft_block_rows) * (op->ft_out / b200::kTileCols);
    return 8LL * op->n * op->nnz * op->ft_out <= (tiles >= 512 ? kGatherMostManyTiles : tiles >= sms ? kGatherMost : tiles >= 16 ? kGatherMostFewTiles : kGatherMostFewestTiles);
}

int finish_op(cudaStream_t stream, const b200_ft_op* op, StatusWord& word, const int* status) {
    int reported = 0;
    if (!word.status) CK(cudaMemcpyAsync(&reported, status, sizeof reported, cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));
    word.finished = true;
    if (word.status) reported = *reinterpret_cast<const volatile int*>(status);
    if (reported & b200::kStatusOutsideBlock)
        return b200::fail(B200_ERR_DATA, "a feature index fell outside the row block of its position (ft_block_rows=%d)", op->ft_block_rows);
    return 0;
}

// Scratch out of the device's pool, for one call.
struct PoolScratch {
    ~PoolScratch() {
        if (at) cudaFreeAsync(at, stream);
    }
    cudaStream_t stream;
    int* at = nullptr;
};

// Groups the pairs into scratch and runs the tiled forward, or the gather forward as it is; synchronises the stream and
// reports a feature outside its block.  `scratch` null: from the pool, if the call needs any; else nothing is allocated.
int run_op(int device, cudaStream_t stream, const b200_ft_op* op, int* scratch) {
    const int n = op->n, R = op->ft_block_rows, nblocks = op->n_inputs / R;
    int sms = 0;
    CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    const bool gathered = few_positions(op, sms);
    PoolScratch own{stream};
    StatusWord word(device, stream);
    if (!scratch && !(gathered && word.status)) {
        if (int rc = b200::op_pool_alloc(device, stream, scratch_ints(n, op->nnz, nblocks) * sizeof(int), &own.at)) return rc;
        scratch = own.at;
    }
    int* status = word.status ? word.status : scratch + kStatusAt;
    b200::FtArgs a{};
    a.table = op->table;
    a.bias = op->bias;
    a.idx_stm = op->idx_stm;
    a.idx_nstm = op->idx_nstm;
    a.n = n;
    a.nnz = op->nnz;
    a.H = op->ft_out;
    a.n_inputs = op->n_inputs;
    a.act = op->ft_act;
    a.x = op->x;
    a.u = op->u;
    if (gathered) {
        a.block_rows = R;
        a.status = status;
        if (!word.status) CK(cudaMemsetAsync(status, 0, sizeof *status, stream));
        const b200::GatherShape g = b200::gather_shape(n, op->pairwise ? a.H / 2 : a.H, op->pairwise, false, sms);
        (op->pairwise ? b200::gather_form<true, false>(g) : b200::gather_form<false, false>(g))<<<g.grid, 256, 0, stream>>>(a, g.pairs);
        CK(cudaGetLastError());
        return finish_op(stream, op, word, status);
    }
    int* begin = scratch;
    int* info = scratch + kScratchHeader;
    int* pairs = info + align_ints((size_t)2 * n);
    int* lists = pairs + align_ints((size_t)4 * n);
    int* hist = lists + (size_t)n * list_len(op->nnz);
    b200::GroupArgs g{};
    g.stm = op->idx_stm;
    g.nstm = op->idx_nstm;
    g.n = n;
    g.nnz = op->nnz;
    g.n_inputs = op->n_inputs;
    g.block_rows = R;
    g.nblocks = nblocks;
    g.n_out_buckets = 1;
    g.info = info;
    g.hist = hist;
    g.status = status;
    g.clear_status = !word.status;
    g.want_lists = 1;
    g.pairs = reinterpret_cast<int2*>(pairs);
    g.lists = reinterpret_cast<uint16_t*>(lists);
    g.list_len = list_len(op->nnz);
    g.block_begin = begin;
    if (nblocks > b200::kGroupMaxBlocks) {
        int *at = hist + nblocks + 1, *spare = at + nblocks + 3;
        CK(cudaMemsetAsync(hist, 0, (size_t)(nblocks + 1) * sizeof(int), stream));
        b200::group_many_count_kernel<<<(2 * n + 7) / 8, 256, 0, stream>>>(g, hist);
        b200::group_many_scan_kernel<<<1, 1024, 0, stream>>>(g, hist, at, spare);
        b200::group_many_place_kernel<<<(2 * n + 7) / 8, 256, 0, stream>>>(g, hist);
    } else {
        const bool vec = b200::group_vec(g);
        b200::group_lists_kernel<<<b200::group_ctas(n), b200::kGroupThreads, 0, stream>>>(g, vec);
        const bool scans = b200::group_scans(n);
        if (scans) CK(b200::launch_step(true, b200::group_scan_kernel, nblocks + 1, 1024, 0, stream, hist, b200::group_ctas(n), nblocks + 1));
        CK(b200::launch_step(true, b200::group_place_kernel, b200::group_windows(n), b200::kPlaceThreads, 0, stream, g, (int)vec, (int)scans));
    }
    CK(cudaGetLastError());

    b200::TileArgs t{};
    t.block_rows = R;
    t.nslabs = op->ft_out / b200::kTileCols;
    t.first_block = 0;
    t.last_block = nblocks;
    t.pairs = g.pairs;
    t.block_begin = begin;
    t.status = status;
    t.lists = g.lists;
    t.list_len = g.list_len;
    t.walk_warps = b200::ft_fwd_warps(R, t.list_len);
    t.fill_steps = (t.block_rows + b200::kFwdThreads / 8 - 1) / (b200::kFwdThreads / 8);
    const size_t smem = b200::ft_fwd_smem(R, t.list_len);
    // one CTA per SM, each taking an equal piece of the (block, slab, pair) work line
    const int ctas = (int)std::max<long long>(1, std::min<long long>(sms, (long long)2 * n * t.nslabs / 128));
    // the caller's arrays may start on any float: pieces of 8 and 16 bytes where they do so, else single floats
    const bool any = (((uintptr_t)op->bias | (uintptr_t)op->x | (op->pairwise ? (uintptr_t)op->u : 0)) & (op->pairwise ? 7 : 15)) != 0;
    const bool ahead = b200::ft_fwd_ahead(a, t, ctas);
    void (*const kernel)(b200::FtArgs, b200::TileArgs) =
        ahead ? (op->pairwise ? (any ? b200::ft_forward_tiled_kernel<true, true, true> : b200::ft_forward_tiled_kernel<true, true, false>)
                              : (any ? b200::ft_forward_tiled_kernel<false, true, true> : b200::ft_forward_tiled_kernel<false, true, false>))
              : (op->pairwise ? (any ? b200::ft_forward_tiled_kernel<true, false, true> : b200::ft_forward_tiled_kernel<true, false, false>)
                              : (any ? b200::ft_forward_tiled_kernel<false, false, true> : b200::ft_forward_tiled_kernel<false, false, false>));
    CK(b200::allow_smem(kernel));
    CK(b200::launch_step(true, kernel, ctas, b200::kFwdThreads, smem, stream, a, t));
    return finish_op(stream, op, word, status);
}

}  // namespace

// One pool per device for the scratch of b200_op_ft_forward (cudaMalloc and cudaFree synchronise the device and cost 0.6 ms and more a
// call; the pool's stream-ordered ones do not).  It keeps at most kPoolKeep bytes between calls, for as long as the
// process lives or until a network that finds no room for its own buffers has it give those back (op_pool_trim).  Stream-ordered, so calls on several streams and
// threads never share memory that is in use.
namespace b200 {
namespace {
constexpr uint64_t kPoolKeep = 32u << 20;
constexpr int kPoolDevices = 64;
std::mutex pool_lock;
cudaMemPool_t pools[kPoolDevices] = {};
}  // namespace

int op_pool_alloc(int device, cudaStream_t stream, size_t bytes, int** out) {
    if (device < 0 || device >= kPoolDevices) return fail(B200_ERR_ARG, "op_ft_forward: device %d out of range", device);
    cudaMemPool_t pool = nullptr;
    {
        std::lock_guard<std::mutex> guard(pool_lock);
        if (!pools[device]) {
            cudaMemPoolProps props{};
            props.allocType = cudaMemAllocationTypePinned;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = device;
            cudaMemPool_t made = nullptr;
            CK(cudaMemPoolCreate(&made, &props));
            uint64_t keep = kPoolKeep;
            CK(cudaMemPoolSetAttribute(made, cudaMemPoolAttrReleaseThreshold, &keep));
            pools[device] = made;
        }
        pool = pools[device];
    }
    void* raw = nullptr;
    CK(cudaMallocFromPoolAsync(&raw, bytes, pool, stream));
    *out = static_cast<int*>(raw);
    return 0;
}

void op_pool_trim(int device) {
    std::lock_guard<std::mutex> guard(pool_lock);
    if (device >= 0 && device < kPoolDevices && pools[device]) cudaMemPoolTrimTo(pools[device], 0);
}
}  // namespace b200

extern "C" {

int b200_op_ft_forward(int device, void* stream, const b200_ft_op* op) {
    if (int rc = check_op(op, "op_ft_forward")) return rc;
    CK(cudaSetDevice(device));
    return run_op(device, static_cast<cudaStream_t>(stream), op, nullptr);
}

// Same result as b200_op_ft_forward without touching the allocator.  It is meant for code
// that shares a GPU with a running training loop, or that runs after the process has handed
// out all of its device memory: cudaMalloc and cudaFree synchronise the whole device and
// serialise on a driver lock, so an evaluation thread that allocated per call would stall the
// trainer's streams every time, and a caller with a fixed memory budget has nothing left to
// allocate from.  Here the grouping scratch is the fixed array above and the call makes no
// cudaMalloc, cudaFree or other allocating call.
//
// The first call on each device looks up the array's device address (one
// cudaGetSymbolAddress, with that device current) and keeps it; make that first call before
// starting any stream capture on the thread.  All calls on one device share the array and it
// keeps the previous call's contents: the counters that must start at zero are cleared at
// the start of every call, and two calls whose GPU work overlaps (different streams or
// threads, same device) would overwrite each other's grouping — run them one after the other.
int b200_op_ft_forward_noalloc(int device, void* stream, const b200_ft_op* op) {
    if (int rc = check_op(op, "op_ft_forward_noalloc")) return rc;
    const int most = op->nnz <= 32 ? B200_OP_NOALLOC_MAX_POSITIONS : B200_OP_NOALLOC_MAX_POSITIONS / 2;
    if (op->n > most || scratch_ints(op->n, op->nnz, op->n_inputs / op->ft_block_rows) > kStaticInts)
        return b200::fail(B200_ERR_ARG,
                          "op_ft_forward_noalloc: %d positions do not fit the fixed scratch, which holds at most %d with "
                          "nnz=%d; split the batch or call b200_op_ft_forward",
                          op->n, most, op->nnz);
    constexpr int kMaxDevices = 64;
    if (device < 0 || device >= kMaxDevices)
        return b200::fail(B200_ERR_ARG, "op_ft_forward_noalloc: device %d out of range", device);
    CK(cudaSetDevice(device));
    // In host code `g_op_scratch` is only a handle for the runtime, not an address a kernel
    // could use: ask once per device, with that device current, where the array lives there.
    static std::mutex lock;
    static int* address[kMaxDevices] = {nullptr};
    int* scratch = nullptr;
    {
        std::lock_guard<std::mutex> guard(lock);
        if (!address[device]) {
            void* p = nullptr;
            CK(cudaGetSymbolAddress(&p, g_op_scratch));
            address[device] = static_cast<int*>(p);
        }
        scratch = address[device];
    }
    return run_op(device, static_cast<cudaStream_t>(stream), op, scratch);
}

}  // extern "C"
