// C-ABI entry points of the linear and embedding path: argument checks and
// kernel selection. Checks mirror the reference wrappers' (_check_packed /
// _check_activations, src/ternel_mlx/kernels.py:1191-1212,1274-1284): shape and
// dtype violations are reported before anything is launched.
#include "tq1_common.cuh"

using namespace tq1;

// A function of the driver, null where there is none.
template <class F>
static F driver_function(const char *name) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &qres) != cudaSuccess || qres != cudaDriverEntryPointSuccess) p = nullptr;
    return reinterpret_cast<F>(p);
}

EncodeTiledFn tq1::encode_tiled_fn() {
    static const EncodeTiledFn fn = driver_function<EncodeTiledFn>("cuTensorMapEncodeTiled");
    return fn;
}

int tq1::device_slot() {
    // asked several times per launch: of the driver where a context is current, which answers sooner than the runtime
    static const auto ask = driver_function<CUresult (*)(CUdevice *)>("cuCtxGetDevice");
    int dev = 0;
    if ((!ask || ask(&dev) != CUDA_SUCCESS) && cudaGetDevice(&dev) != cudaSuccess) return 0;
    return dev >= 0 && dev < kMaxDevices ? dev : 0;
}

int tq1::sm_count() {
    static std::atomic<int> count[kMaxDevices];
    const int dev = device_slot();
    int n = count[dev].load(std::memory_order_relaxed);
    if (!n) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        count[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

cudaError_t tq1::opt_in(KernelRecord &record, const void *kernel, size_t smem, bool large_clusters) {
    std::atomic<bool> &done = record.opted_in[device_slot()];
    if (done.load(std::memory_order_acquire)) return cudaSuccess;
    cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err == cudaSuccess && large_clusters) err = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (err == cudaSuccess) done.store(true, std::memory_order_release);
    return err;
}

// What is made of the driver's answer: it says 0 of a size that this device cannot run, and nothing on a machine without one, where
// calls are planned only.
static int cluster_count(bool answered, int n, bool device, int size) {
    static const int of_b200[kMaxCluster + 1] = {0, 148, 74, 45, 33, 26, 22, 15, 15, 14, 14, 8, 8, 8, 8, 8, 8};
    return answered ? n : device ? 0 : of_b200[size];
}

int tq1::clusters_at_once(KernelRecord &record, const void *kernel, unsigned threads, size_t smem, int size) {
    if (size == 1) return sm_count();
    std::atomic<int> &known = record.clusters[device_slot()][size];
    int n = known.load(std::memory_order_relaxed);
    if (!n) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(sm_count() / size * size));
        cfg.blockDim = dim3(threads);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = (unsigned)size;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        if (size > 8) cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        const bool answered = opt_in(record, kernel, smem) == cudaSuccess && cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess;
        int devices = 0;
        if (!answered) {
            cudaGetLastError();
            if (cudaGetDeviceCount(&devices) != cudaSuccess) { cudaGetLastError(); devices = 0; }
        }
        n = cluster_count(answered, n, devices > 0, size);
        if (n < 1) n = -1;                                      // known to be none
        known.store(n, std::memory_order_relaxed);
    }
    return n > 0 ? n : 0;
}

namespace {

struct GraphTail { unsigned long long capture; cudaGraphNode_t node; };
// The last kernel of this library that this thread has captured: in which capture, which node.
thread_local GraphTail t_own = {};

// The node that the next one captured on the stream will depend on, if there is one such.
GraphTail tail_of(cudaStream_t stream) {
    GraphTail tail = {};
    cudaStreamCaptureStatus status;
    const cudaGraphNode_t *nodes = nullptr;
    const cudaGraphEdgeData *edges = nullptr;
    size_t n = 0;
    if (cudaStreamGetCaptureInfo_v3(stream, &status, &tail.capture, nullptr, &nodes, &edges, &n) != cudaSuccess) cudaGetLastError();
    else if (n == 1) tail.node = nodes[0];
    return tail;
}

}  // namespace

// Whether the stream is being captured. Asked by every launch, so of the driver, which answers in 17 ns (the runtime in 46).
bool tq1::stream_captured(cudaStream_t stream) {
    static const auto ask = driver_function<CUresult (*)(CUstream, CUstreamCaptureStatus *)>("cuStreamIsCapturing");
    CUstreamCaptureStatus status = CU_STREAM_CAPTURE_STATUS_NONE;
    return ask && ask(stream, &status) == CUDA_SUCCESS && status == CU_STREAM_CAPTURE_STATUS_ACTIVE;
}

bool tq1::behind_own_kernel(cudaStream_t stream) {
    const GraphTail tail = tail_of(stream);
    return tail.node && tail.capture == t_own.capture && tail.node == t_own.node;
}

void tq1::note_captured_kernel(cudaStream_t stream) { t_own = tail_of(stream); }

// Bytes that a call of this shape uses.
static size_t linear_scratch_bytes(int M, int N, int K) {
    if (M <= 0 || N <= 0 || K <= 0 || K % kGroup) return 0;
    if (M == 1 && gemv_chain_shape_ok(N, K)) return gemv_chain_workspace_bytes(N, K);
    if (gemm_tc_shape_ok(M, N, K)) return gemm_tc_workspace_bytes(M, N, K);
    // the kernel for the other widths runs without a workspace; a caller that has one finds its status word in place
    return gemm_groups_preferred(M, N, K) ? kWsStatusBytes : 0;
}

extern "C" {

// Bytes that calls of this shape and of every smaller one with K % 512 == 0 use: how many partial tiles a shape leaves does
// not grow with it (257 tokens take tiles of 144, 256 tokens a tile of 256), but callers make one workspace for the largest.
size_t tq1_linear_workspace_bytes(int M, int N, int K) {
    const size_t used = linear_scratch_bytes(M, N, K);
    if (used == 0 || K % 512) return used;
    return M == 1 ? gemv_chain_workspace_bound(N, K) : gemm_tc_workspace_bound(M);
}

int tq1_linear_f16(const uint8_t *blocks, const void *x, void *y, int y_is_f32,
                   int M, int N, int K, void *workspace, size_t workspace_bytes, void *stream) {
    if (!blocks || !x || !y) return fail(TQ1_ERR_INVALID, "tq1_linear_f16: null pointer");
    if (M <= 0) return fail(TQ1_ERR_INVALID, "activations have an empty batch dimension");
    if (N <= 0 || K <= 0)
        return fail(TQ1_ERR_INVALID, "tensor dimensions must be positive, got %dx%d", N, K);
    if (K % kGroup)
        return fail(TQ1_ERR_INVALID, "%d columns is not a multiple of the 128-weight group", K);
    if (reinterpret_cast<uintptr_t>(blocks) & 3)
        return fail(TQ1_ERR_INVALID, "tq1_linear_f16: blocks must be 4-byte aligned");
    if (reinterpret_cast<uintptr_t>(x) & 15)
        return fail(TQ1_ERR_INVALID, "tq1_linear_f16: x must be 16-byte aligned");
    const size_t need = linear_scratch_bytes(M, N, K);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (need && K % 512 == 0 && (!workspace || workspace_bytes < need || (reinterpret_cast<uintptr_t>(workspace) & 255)))
        return fail(TQ1_ERR_WORKSPACE, "tq1_linear_f16: workspace of %zu bytes (256-byte aligned) required", need);
    if (M == 1 && gemv_chain_fits(blocks, N, K))
        return launch_gemv_single(blocks, static_cast<const __half *>(x), y, y_is_f32 != 0, N, K, false, workspace,
                                  kWsSlotRegionBytes, s);
    int status = TQ1_OK;
    if (need >= kWsScratchOffset &&
        try_gemv_looped(blocks, static_cast<const __half *>(x), y, y_is_f32 != 0, M, N, K, false, workspace, s, &status))
        return status;
    if ((reinterpret_cast<uintptr_t>(blocks) & 15) == 0 &&
        try_gemm_slices(blocks, static_cast<const __half *>(x), y, y_is_f32 != 0, M, N, K, workspace, s, false, &status))
        return status;
    if ((reinterpret_cast<uintptr_t>(blocks) & 15) == 0 && gemm_tc_shape_ok(M, N, K))
        return launch_gemm_tc(blocks, static_cast<const __half *>(x), y, y_is_f32 != 0, M, N, K, workspace, s);
    if (gemm_groups_preferred(M, N, K)) {
        unsigned *word = workspace && workspace_bytes >= kWsStatusBytes && (reinterpret_cast<uintptr_t>(workspace) & 3) == 0
                             ? static_cast<unsigned *>(workspace) : nullptr;
        return launch_gemm_groups(gemm_groups_form(M, N, K, word != nullptr), blocks, static_cast<const __half *>(x), y,
                                  y_is_f32 != 0, M, N, K, word, s);
    }
    return launch_gemv_rows(blocks, static_cast<const __half *>(x), y, y_is_f32 != 0, M, N, K, s);
}

int tq1_linear_swiglu_f16(const uint8_t *blocks, const void *x, void *y, int y_is_f32, int M, int N, int K,
                          void *workspace, size_t workspace_bytes, void *stream) {
    if (!blocks || !x || !y) return fail(TQ1_ERR_INVALID, "tq1_linear_swiglu_f16: null pointer");
    if (M <= 0) return fail(TQ1_ERR_INVALID, "activations have an empty batch dimension");
    if (N <= 0 || K <= 0) return fail(TQ1_ERR_INVALID, "tensor dimensions must be positive, got %dx%d", N, K);
    if (N > (1 << 30)) return fail(TQ1_ERR_INVALID, "tq1_linear_swiglu_f16: too many rows");
    const int rows = 2 * N;                 // (gate, up) pairs
    if (reinterpret_cast<uintptr_t>(x) & 15)
        return fail(TQ1_ERR_INVALID, "tq1_linear_swiglu_f16: x must be 16-byte aligned");
    const __half *xh = static_cast<const __half *>(x);
    const bool gemv = M == 1 && gemv_chain_fits(blocks, rows, K);
    if (!gemv && (M < 2 || K % 512 || (reinterpret_cast<uintptr_t>(blocks) & 15)))
        return fail(TQ1_ERR_INVALID,
                    "tq1_linear_swiglu_f16: needs K %% 512 == 0 and 16-byte aligned blocks (got %dx%d)", rows, K);
    const size_t need = linear_scratch_bytes(M, rows, K);
    if (!workspace || workspace_bytes < need || (reinterpret_cast<uintptr_t>(workspace) & 255))
        return fail(TQ1_ERR_WORKSPACE, "tq1_linear_swiglu_f16: workspace of %zu bytes (256-byte aligned) required", need);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (gemv) return launch_gemv_single(blocks, xh, y, y_is_f32 != 0, rows, K, true, workspace, kWsSlotRegionBytes, s);
    int status = TQ1_OK;
    if (try_gemv_looped(blocks, xh, y, y_is_f32 != 0, M, rows, K, true, workspace, s, &status)) return status;
    if (try_gemm_slices(blocks, xh, y, y_is_f32 != 0, M, rows, K, workspace, s, true, &status)) return status;
    return launch_gemm_tc(blocks, xh, y, y_is_f32 != 0, M, rows, K, workspace, s, true);
}

int tq1_linear_plan(int M, int N, int K, int aligned, int *kernel, int *token_tile, int *ctas, int *parts) {
    if (!kernel || !token_tile || !ctas || !parts) return fail(TQ1_ERR_INVALID, "tq1_linear_plan: null pointer");
    if (M <= 0 || N <= 0 || K <= 0 || K % kGroup) return fail(TQ1_ERR_INVALID, "tq1_linear_plan: bad shape");
    *token_tile = *ctas = *parts = 0;
    if (aligned && (M == 1 ? gemv_chain_shape_ok(N, K) : gemv_looped_shape_ok(M, N, K))) {
        *kernel = TQ1_KERNEL_STREAM_GEMV;       // the tile kernel or the chain kernel
    } else if (aligned && gemm_tc_shape_ok(M, N, K)) {
        *kernel = TQ1_KERNEL_TENSOR_CORE;
        gemm_tc_plan(M, N, K, token_tile, ctas, parts);
    } else if (gemm_groups_preferred(M, N, K)) {
        *kernel = TQ1_KERNEL_GROUP_SUMS;
    } else {
        *kernel = TQ1_KERNEL_ROWS;
    }
    return TQ1_OK;
}

int tq1_linear_form(int M, int N, int K, int aligned, int has_workspace, int *form) {
    int kernel, token_tile, ctas, parts;
    if (!form) return fail(TQ1_ERR_INVALID, "tq1_linear_form: null pointer");
    const int rc = tq1_linear_plan(M, N, K, aligned, &kernel, &token_tile, &ctas, &parts);
    if (rc != TQ1_OK) return rc;
    *form = kernel == TQ1_KERNEL_TENSOR_CORE   ? (gemm_slices_preferred(M, N, K) ? TQ1_FORM_SLICES : TQ1_FORM_TCGEN05)
            : kernel == TQ1_KERNEL_GROUP_SUMS  ? gemm_groups_form(M, N, K, has_workspace != 0)
            : kernel == TQ1_KERNEL_STREAM_GEMV ? TQ1_FORM_STREAM_GEMV
                                               : TQ1_FORM_ROWS;
    return TQ1_OK;
}

// Sweep recording only (ternel_b200/dispatch.py binds it by name): forces the tensor-core kernel's token tile
// for every later call of this process; 0 restores the rule. Process-global and not thread-safe, which is why
// it is not part of the public header.
// Sweep recording only: the largest batch that runs as passes of the batch-1 kernel (0: none).
int tq1_debug_set_loop_tokens(int tokens) {
    if (gemv_set_loop_tokens(tokens) != TQ1_OK)
        return fail(TQ1_ERR_INVALID, "tq1_debug_set_loop_tokens: %d is not in 0..8", tokens);
    return TQ1_OK;
}

// Sweep recording only: the product by one of the forms that share calls between them (TQ1_FORM_SLICES with K % 512 == 0 and
// aligned blocks, or one of the group sums), whichever the rules would take. Arguments as those of tq1_linear_f16, checked less.
int tq1_debug_linear_as(int form, const uint8_t *blocks, const void *x, void *y, int y_is_f32, int M, int N, int K,
                        void *workspace, void *stream) {
    if (!blocks || !x || !y || !workspace || M <= 0 || N <= 0 || K <= 0 || K % kGroup)
        return fail(TQ1_ERR_INVALID, "tq1_debug_linear_as: bad call");
    const __half *xh = static_cast<const __half *>(x);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (form == TQ1_FORM_SLICES && K % 512 == 0 && M >= 3 && M <= 16 && (reinterpret_cast<uintptr_t>(blocks) & 15) == 0)
        return launch_gemm_slices(blocks, xh, y, y_is_f32 != 0, M, N, K, workspace, s);
    if (form >= TQ1_FORM_GROUPS_FEW && form <= TQ1_FORM_GROUPS_TCGEN05 && M >= 2)
        return launch_gemm_groups(form, blocks, xh, y, y_is_f32 != 0, M, N, K, static_cast<unsigned *>(workspace), s);
    return fail(TQ1_ERR_INVALID, "tq1_debug_linear_as: form %d does not take %dx%dx%d", form, M, N, K);
}

// Tests only: the layout of a call by the kernel of `form` (TQ1_FORM_STREAM_GEMV: one or two activation rows as a call of their own;
// TQ1_FORM_SLICES; TQ1_FORM_TCGEN05, whose sets are the parts of a tile, and which has no ring stages here), whether or not the rules
// would send it there. layout: CTAs of a cluster, sets of warps, ring stages, row tiles of a cluster, and whether the rules do. All
// zero: it does not fit that kernel.
int tq1_debug_call_layout(int form, int M, int N, int K, const int *rooms, int *layout) {
    if (!layout || M <= 0 || N <= 0 || K <= 0 || K % kGroup) return fail(TQ1_ERR_INVALID, "tq1_debug_call_layout: bad call");
    CallLayout l = {};
    if (form == TQ1_FORM_STREAM_GEMV) {
        if (!gemv_tiles_layout(M, N, K, rooms, &l)) l = {};
    } else if (form == TQ1_FORM_SLICES) {
        if (!gemm_slices_layout(M, N, K, rooms, &l)) l = {};
    } else if (form == TQ1_FORM_TCGEN05) {
        if (!gemm_tc_layout(M, N, K, rooms, &l)) l = {};
    } else {
        return fail(TQ1_ERR_INVALID, "tq1_debug_call_layout: form %d", form);
    }
    layout[0] = l.cluster;
    layout[1] = l.sets;
    layout[2] = l.stages;
    layout[3] = l.tiles;
    layout[4] = l.preferred;
    return TQ1_OK;
}

// Tests only.
int tq1_debug_cluster_count(int answered, int n, int device, int size) { return cluster_count(answered != 0, n, device != 0, size); }

int tq1_debug_force_token_tile(int token_tile) {
    if (gemm_tc_force_tile(token_tile) != TQ1_OK)
        return fail(TQ1_ERR_INVALID, "tq1_debug_force_token_tile: %d is not 0, 16, 32, 64, 128 or 256", token_tile);
    return TQ1_OK;
}

static size_t shard_local_bytes(int M, int N_local) {
    return ((size_t)M * N_local * sizeof(__half) + 255) & ~(size_t)255;
}

size_t tq1_linear_sharded_workspace_bytes(int M, int N_local, int K) {
    size_t base = tq1_linear_workspace_bytes(M, N_local, K);
    if (base < kWsScratchOffset) base = kWsScratchOffset;
    base = (base + 255) & ~(size_t)255;
    return base + shard_local_bytes(M, N_local);
}

int tq1_shard_advance_epoch(uint32_t *epoch_base, uint32_t delta, void *stream) {
    if (!epoch_base) return fail(TQ1_ERR_INVALID, "tq1_shard_advance_epoch: null pointer");
    return launch_epoch_advance(epoch_base, delta, static_cast<cudaStream_t>(stream));
}

int tq1_linear_f16_sharded(const uint8_t *blocks, const void *x, const tq1_shard *shard, int M, int N_local, int K,
                           void *workspace, size_t workspace_bytes, void *stream) {
    if (!blocks || !x || !shard) return fail(TQ1_ERR_INVALID, "tq1_linear_f16_sharded: null pointer");
    if (shard->world < 1 || shard->world > kMaxRanks || shard->rank < 0 || shard->rank >= shard->world)
        return fail(TQ1_ERR_INVALID, "tq1_linear_f16_sharded: rank %d of %d is out of range (at most %d ranks)",
                    shard->rank, shard->world, kMaxRanks);
    if (M <= 0) return fail(TQ1_ERR_INVALID, "activations have an empty batch dimension");
    if (N_local <= 0 || K <= 0 || K % kGroup)
        return fail(TQ1_ERR_INVALID, "tq1_linear_f16_sharded: bad shard shape %dx%d", N_local, K);
    if (N_local % kFlagRows)
        return fail(TQ1_ERR_INVALID, "tq1_linear_f16_sharded: a shard of %d rows is not a multiple of %d", N_local,
                    kFlagRows);
    if (shard->wait_flags && shard->wait_tiles < 0)
        return fail(TQ1_ERR_INVALID, "tq1_linear_f16_sharded: negative wait_tiles");
    if (shard->n_offset < 0 || shard->n_offset % 16 || shard->n_offset + N_local > shard->n_total)
        return fail(TQ1_ERR_INVALID, "tq1_linear_f16_sharded: rows [%d, %d) do not fit %d gathered rows "
                    "(the offset must be a multiple of 16)", shard->n_offset, shard->n_offset + N_local, shard->n_total);
    const size_t need = tq1_linear_sharded_workspace_bytes(M, N_local, K);
    if (!workspace || workspace_bytes < need || (reinterpret_cast<uintptr_t>(workspace) & 255))
        return fail(TQ1_ERR_WORKSPACE, "tq1_linear_f16_sharded: workspace of %zu bytes (256-byte aligned) required", need);
    ShardDev sd = {};
    sd.world = shard->world;
    sd.rank = shard->rank;
    for (int p = 0; p < shard->world; ++p) {
        if (!shard->peer_y[p] || !shard->peer_flags[p])
            return fail(TQ1_ERR_INVALID, "tq1_linear_f16_sharded: missing peer pointer for rank %d", p);
        sd.peer_y[p] = static_cast<__half *>(shard->peer_y[p]) + shard->n_offset;
        sd.peer_flags[p] = shard->peer_flags[p] + shard->n_offset / kFlagRows;
    }
    sd.epoch_base = shard->epoch_base;
    sd.publish_epoch = shard->publish_epoch;
    sd.wait_flags = shard->wait_flags;
    sd.wait_tiles = shard->wait_flags ? shard->wait_tiles : 0;
    sd.wait_epoch = shard->wait_epoch;
    sd.ld_total = shard->n_total;
    unsigned *status = static_cast<unsigned *>(workspace);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // wait for the inputs, compute the local slice, push it
    int rc = launch_shard_wait(sd, status, s);
    if (rc != TQ1_OK) return rc;
    const size_t base = need - shard_local_bytes(M, N_local);
    __half *local = reinterpret_cast<__half *>(static_cast<unsigned char *>(workspace) + base);
    rc = tq1_linear_f16(blocks, x, local, 0, M, N_local, K, workspace, base, stream);
    if (rc != TQ1_OK) return rc;
    return launch_shard_push(local, M, N_local, sd, s);
}

int tq1_gemv_f16_noalloc(const uint8_t *blocks, const void *x, void *y, int y_is_f32, int N, int K, void *stream) {
    if (!blocks || !x || !y) return fail(TQ1_ERR_INVALID, "tq1_gemv_f16_noalloc: null pointer");
    if (N <= 0 || K <= 0)
        return fail(TQ1_ERR_INVALID, "tensor dimensions must be positive, got %dx%d", N, K);
    if (K % kGroup)
        return fail(TQ1_ERR_INVALID, "%d columns is not a multiple of the 128-weight group", K);
    if (reinterpret_cast<uintptr_t>(x) & 15)
        return fail(TQ1_ERR_INVALID, "tq1_gemv_f16_noalloc: x must be 16-byte aligned");
    return gemv_noalloc(blocks, static_cast<const __half *>(x), y, y_is_f32 != 0, N, K,
                        static_cast<cudaStream_t>(stream));
}

int tq1_gemv_noalloc_status(uint32_t *status_host, void *stream) {
    if (!status_host) return fail(TQ1_ERR_INVALID, "tq1_gemv_noalloc_status: null pointer");
    return gemv_noalloc_status(status_host, static_cast<cudaStream_t>(stream));
}

int tq1_embedding_f16(const uint8_t *blocks, const int64_t *ids, void *out, int out_is_f32,
                      int64_t T, int64_t V, int K, void *stream) {
    if (!blocks || !ids || !out) return fail(TQ1_ERR_INVALID, "tq1_embedding_f16: null pointer");
    if (T <= 0) return fail(TQ1_ERR_INVALID, "indices are empty");
    if (V <= 0 || K <= 0)
        return fail(TQ1_ERR_INVALID, "tensor dimensions must be positive, got %lldx%d", (long long)V, K);
    if (K % kGroup)
        return fail(TQ1_ERR_INVALID, "%d columns is not a multiple of the 128-weight group", K);
    if (reinterpret_cast<uintptr_t>(blocks) & 3)
        return fail(TQ1_ERR_INVALID, "tq1_embedding_f16: blocks must be 4-byte aligned");
    if (reinterpret_cast<uintptr_t>(out) & 15)
        return fail(TQ1_ERR_INVALID, "tq1_embedding_f16: out must be 16-byte aligned");
    return launch_embedding(blocks, ids, out, out_is_f32 != 0, T, V, K, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
