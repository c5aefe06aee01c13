// The whole kNN forward as one host call: build, status word, search and the copy of the cell order.
//
// Small batches are bound by the host.  A caller in an interpreter pays for every call into the
// library and for the event and the pinned word of the status check; here they cost one call, and the
// wait for the status word happens without the interpreter (two row splits of 5000 points, K = 16, forward and
// backward, B200, timed in turn: 196 -> 168 us; a GravNet layer on ten small events: 303 -> 289 us;
// with the build in one launch and the words looked for 128 and 240 since).
#include <mutex>
#include <thread>

#include "knn_tree.cuh"

namespace fgc {

// Two page-locked words, mapped on every device, and an event of one device.  A call that waits takes a slot of its own
// for the time of the wait and gives it back, so any number of threads and streams may call at once.  Slots are shared
// by all threads: a thread that ends frees nothing (freeing page-locked memory may wait for the device, and breaks another
// thread's graph capture).  At most kKeptSlots stay for later calls, i.e. 4 KB.
struct StatusSlot {
    int32_t *words = nullptr;          // written as one
    cudaEvent_t ready = nullptr;
    int device = -1;
};
constexpr size_t kKeptSlots = 64;
constexpr int64_t kNoWords = -1;               // (a status has no sign)

struct StatusPool {
    std::mutex lock;
    StatusSlot kept[kKeptSlots];
    size_t n = 0;
};

static StatusPool &status_pool()
{
    static StatusPool *pool = new StatusPool;      // never destroyed: threads may outlive static objects
    return *pool;
}

// Allocations, and queries of an event, that are harmless to a graph capture of another thread.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

static void free_slot(StatusSlot &s)
{
    const RelaxedCapture relaxed;
    if (s.ready) cudaEventDestroy(s.ready);
    if (s.words) cudaFreeHost(s.words);
    s = StatusSlot();
}

static cudaError_t take_slot(StatusSlot &s)
{
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    {
        StatusPool &pool = status_pool();
        const std::lock_guard<std::mutex> hold(pool.lock);
        for (size_t i = pool.n; i-- > 0;)
            if (pool.kept[i].device == device) {
                s = pool.kept[i];
                pool.kept[i] = pool.kept[--pool.n];
                return cudaSuccess;
            }
    }
    const RelaxedCapture relaxed;
    s.device = device;
    e = cudaHostAlloc((void **)&s.words, 64, cudaHostAllocPortable | cudaHostAllocMapped);
    if (e != cudaSuccess) s.words = nullptr;
    else e = cudaEventCreateWithFlags(&s.ready, cudaEventDisableTiming);
    if (e != cudaSuccess) free_slot(s);
    return e;
}

static void give_back(StatusSlot &s)
{
    {
        StatusPool &pool = status_pool();
        const std::lock_guard<std::mutex> hold(pool.lock);
        if (pool.n < kKeptSlots) {
            pool.kept[pool.n++] = s;
            return;
        }
    }
    free_slot(s);
}

static int knn_forward_launch(const float *coords, int64_t n_vert, int32_t n_coords, const int64_t *row_splits, int64_t n_rs,
                              int32_t K, const int64_t *direction, int32_t tf_compat, float target_occupancy, int32_t flags,
                              int64_t *out_idx, float *out_distsq, int32_t *out_order, void *ws, size_t ws_bytes,
                              const StatusSlot *status, bool *published, fgc_stream_t stream)
{
    const bool tree = (flags & FGC_FORWARD_TREE) != 0;
    int rc;
    bool words = false, order = tree;      // status words and cell order are written by the build
    if (tree)
        rc = knn_build_tree_forward(coords, n_vert, n_coords, row_splits, n_rs, K, direction, status ? status->words : nullptr, out_order, &words, ws,
                                    ws_bytes, stream);
    else {
        const int dims = flags & FGC_SEARCH_GRID3 ? 3 : (flags & FGC_SEARCH_GRID4 ? 4 : 0);
        rc = knn_build_grid_forward(coords, n_vert, n_coords, row_splits, n_rs, K, direction, target_occupancy, dims,
                                    status ? status->words : nullptr, out_order, &words, ws, ws_bytes, stream);
        order = words;
    }
    if (rc != FGC_OK) return rc;
    if (status) {
        if (!words) rc = fgc_knn_publish_grid_info(ws, status->words, stream);
        if (rc != FGC_OK) return rc;
        *published = true;
        FGC_RETURN_IF_CUDA(cudaEventRecord(status->ready, (cudaStream_t)stream));
    }
    // all queries of a leaf at once, in workspaces with room for its scratch
    bool groups = false;
    if (tree && n_vert > 0 && n_coords <= kGroupDims) {
        const KnnWorkspace L = knn_workspace_layout(n_vert, n_coords, n_rs, K);
        groups = ws_bytes >= L.total + tree_extra_bytes(n_vert, n_coords, n_rs) && tree_layout(L, n_vert, n_coords, n_rs).groups;
    }
    const bool ties = tree && (flags & FGC_FORWARD_GRID_TIES) != 0;
    const TieMarks marks = !ties ? TieMarks::kNone : (flags & FGC_FORWARD_GRID_ORDER ? TieMarks::kAny : TieMarks::kKth);
    if (groups) rc = knn_search_tree_groups(n_vert, n_coords, row_splits, n_rs, K, direction != nullptr, tf_compat, marks, out_idx,
                                            out_distsq, ws, ws_bytes, stream);
    else if (tree) rc = knn_search_tree(n_vert, n_coords, row_splits, n_rs, K, direction != nullptr, tf_compat, marks, out_idx,
                                   out_distsq, ws, ws_bytes, stream);
    else rc = fgc_knn_search(n_vert, n_coords, n_rs, K, direction != nullptr, tf_compat,
                             (flags & (FGC_SEARCH_COUNT | FGC_SEARCH_GRID3 | FGC_SEARCH_GRID4)) | FGC_SEARCH_FRESH, out_idx,
                             out_distsq, ws, ws_bytes, stream);
    if (rc != FGC_OK) return rc;
    if (out_order && n_vert > 0 && !order)
        FGC_RETURN_IF_CUDA(cudaMemcpyAsync(out_order, fgc_knn_cell_order(ws, n_vert, n_coords, n_rs, K),
                                           sizeof(int32_t) * (size_t)n_vert, cudaMemcpyDeviceToDevice, (cudaStream_t)stream));
    if (ties && n_vert > 0) {
        // Which of several points at exactly the K-th distance is kept is open, but for coordinates without order it should
        // not hang on the choice of the search: the few such rows are searched again on a grid.  On a lattice, where
        // nearly every row has such a choice, that would be the whole search twice: beyond a sixteenth of the rows the
        // tree's choice stands.  With FGC_FORWARD_GRID_ORDER rows with equal distances inside the list are among them, or left out where they make
        // the rows too many (4 % of the points twice, K = 65: three rows in four).
        rc = knn_build_grid_for_ties(coords, n_vert, n_coords, row_splits, n_rs, K, direction, target_occupancy, ws, ws_bytes,
                                     stream);
        if (rc != FGC_OK) return rc;
        return knn_search_grid(n_vert, n_coords, n_rs, K, direction != nullptr, tf_compat, FGC_SEARCH_FRESH, true, out_idx,
                               out_distsq, ws, ws_bytes, stream);
    }
    return FGC_OK;
}

}  // namespace fgc

extern "C" int fgc_knn_forward(const float *coords, int64_t n_vert, int32_t n_coords, const int64_t *row_splits,
                               int64_t n_rs, int32_t K, const int64_t *direction_or_null, int32_t tf_compat,
                               float target_occupancy, int32_t flags, int64_t *out_idx, float *out_distsq,
                               int32_t *out_order_or_null, void *workspace, size_t workspace_bytes,
                               int32_t *info_host_or_null, fgc_stream_t stream)
{
    using namespace fgc;
    if (!info_host_or_null)
        return knn_forward_launch(coords, n_vert, n_coords, row_splits, n_rs, K, direction_or_null, tf_compat, target_occupancy,
                                  flags, out_idx, out_distsq, out_order_or_null, workspace, workspace_bytes, nullptr, nullptr,
                                  stream);
    StatusSlot slot;
    FGC_RETURN_IF_CUDA(take_slot(slot));
    *(volatile int64_t *)slot.words = kNoWords;
    bool published = false;
    int rc = knn_forward_launch(coords, n_vert, n_coords, row_splits, n_rs, K, direction_or_null, tf_compat, target_occupancy,
                                flags, out_idx, out_distsq, out_order_or_null, workspace, workspace_bytes, &slot, &published,
                                stream);
    if (!published) {
        give_back(slot);
        return rc;
    }
    // The words are on their way (also after an error of a later launch), and here long before the build has ended: looked for until the
    // event behind the build says that it has.
    const RelaxedCapture relaxed;          // (a query of an event would end another thread's capture)
    volatile int64_t *const words = (volatile int64_t *)slot.words;
    cudaError_t e = cudaErrorNotReady;
    for (int i = 1; *words == kNoWords && e == cudaErrorNotReady; i++)
        if (i % 1024 == 0) {
            if (i > 1 << 17) std::this_thread::yield();
            e = cudaEventQuery(slot.ready);
        }
    if (*words == kNoWords && rc == FGC_OK) rc = e == cudaSuccess ? (int)cudaErrorUnknown : (int)e;
    if (rc == FGC_OK) {
        info_host_or_null[0] = (int32_t)*words;
        info_host_or_null[1] = (int32_t)(*words >> 32);
    }
    // after an error the event may not stand for these words: the slot is not used again
    if (rc == FGC_OK) give_back(slot);
    return rc;
}
