// Shared constants and helpers for the TQ1_G128 kernels (sm_100a).
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "../../include/ternel_b200.h"

namespace tq1 {

constexpr int kGroup = TQ1_GROUP;             // weights per block
constexpr int kBlockBytes = TQ1_BLOCK_BYTES;  // bytes per block
constexpr int kBlockWords = kBlockBytes / 4;  // 7 x 32-bit words, always 4-byte aligned
constexpr int kCodeBytes = 26;
constexpr int kFullBytes = 25;
constexpr int kMaxFull = 242;
constexpr int kMaxTail = 26;

// Workspace layout shared by every linear kernel: [control words, 256 B][partial-sum slots of the
// batch-1 kernel, 16 MiB][counters of the batched kernel, 4 KiB][scratch of the batched
// kernel, or the hand-off words of a chain]. Slots carry sequence tags, so nothing in the slot region ever
// has to be cleared, and the counters are zero between calls; no other kernel writes to either, so calls of
// any shape and kind can share one workspace. The workspace must be zero-filled once before its first use.
constexpr size_t kWsStatusBytes = 256;
constexpr size_t kWsCounterBytes = 4096;
constexpr size_t kWsSlotRegionBytes = (size_t)16 << 20;       // 2^21 slots: 131072 rows of 8192 columns are one link
constexpr size_t kWsCounterOffset = kWsStatusBytes + kWsSlotRegionBytes;
constexpr size_t kWsScratchOffset = kWsCounterOffset + kWsCounterBytes;

// Checked build (-DTQ1_BOUNDS_CHECK -rdc=true): every global store of a kernel (and the reads of scratch that
// other CTAs write) first tests its index against the extent the launcher knows. A violation is counted in
// g_tq1_bounds {count, code of the first, its index, its limit} and the access is SKIPPED: the kernel neither
// traps nor touches memory it does not own. The reference's analogue is the SAFE build of its Metal kernels,
// which clamps row indices (src/ternel_mlx/kernels.py:23-27). tq1_debug_bounds() reads the record.
// Codes: 1x chain kernel (10 slot store, 11 slot read, 12 y, 13 hand-off store, 14 hand-off read),
// 2x row kernel, 3x gather, 4x batched kernel (40 result, 41 partial tile), 5x panels, 6x shard push,
// 7x group sums, 8x slice kernel, 9x tile kernel.
#ifdef TQ1_BOUNDS_CHECK
extern __device__ unsigned long long g_tq1_bounds[4];
__device__ __forceinline__ bool tq1_in_bounds(long long index, long long limit, unsigned code) {
    if (index >= 0 && index < limit) return true;
    if (atomicAdd(&g_tq1_bounds[0], 1ull) == 0ull) {
        g_tq1_bounds[1] = code;
        g_tq1_bounds[2] = (unsigned long long)index;
        g_tq1_bounds[3] = (unsigned long long)limit;
    }
    return false;
}
#define TQ1_IN_BOUNDS(index, limit, code) tq1_in_bounds((long long)(index), (long long)(limit), (code))
#else
#define TQ1_IN_BOUNDS(index, limit, code) true
#endif

// Records a message for tq1_last_error() and returns `code`.
int fail(int code, const char *fmt, ...);
int cuda_fail(cudaError_t err, const char *what);

// cuTensorMapEncodeTiled, looked up once (a thread that comes while another one is looking waits for it); null if unavailable.
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled_fn();

// What launches keep per device: the SM count differs between devices, and the shared-memory opt-in is an attribute of a
// function on one device. A record is filled by whoever comes first; threads that come together write the same.
constexpr int kMaxDevices = 64;
int device_slot();                                      // the current device's
int sm_count();                                         // the current device's, 148 on a machine without one (planning)
constexpr int kMaxCluster = 16;                         // more than eight CTAs are asked for by name (large_clusters)
struct KernelRecord {
    std::atomic<bool> opted_in[kMaxDevices];
    std::atomic<int> clusters[kMaxDevices][kMaxCluster + 1];      // of so many CTAs that run at once
};
// The kernel may have `smem` bytes of dynamic shared memory.
cudaError_t opt_in(KernelRecord &record, const void *kernel, size_t smem, bool large_clusters = false);
// Clusters of `size` CTAs of a kernel that run at the same time: fewer than SMs / CTAs where the SMs of a GPC are no
// multiple of it (with one CTA per SM 74 of 2, 33 of 4 and 15 of 8 on this part); 0 where none does.
int clusters_at_once(KernelRecord &record, const void *kernel, unsigned threads, size_t smem, int size);

// A launch may begin while the kernel before it in the stream ends (programmatic dependent launch): that kernel lets it in
// (allow_next_grid), and it calls grid_dependency_wait() before it touches what an earlier one may have written or may still
// read, by plain loads: __ldg and __restrict__ tell the compiler that the data were there from the kernel's beginning. Calls back
// to back through the Python modules: a gather of 2048 rows of 5120 columns 8.2 -> 5.5 us, five tokens of 4099x2176 7.2 -> 5.9.
//
// Not in a graph behind a kernel that is not this library's and lets nothing in: there the edge alone costs some 0.3 us and up
// to 0.7 (512 rows gathered 3.1 us as an ordinary launch, 3.4 as a dependent one; five tokens of 4099x2176 6.3 and 6.9). Outside
// a graph such a launch gains all the same: the launch itself is brought forward (the gather 4.1 -> 3.1).
bool stream_captured(cudaStream_t stream);              // is being captured; asked once per launch
bool behind_own_kernel(cudaStream_t stream);            // the node that the next one captured depends on is one that was noted
void note_captured_kernel(cudaStream_t stream);         // a kernel of this library that lets the next one in has been captured

// `dependent` where overlapping is asked for (by calls of a stream, by captured ones) and pays, else `plain`, its form for an
// ordinary launch. lets_in: it calls allow_next_grid().
template <class... P, class... A>
cudaError_t launch_either(bool in_stream, bool in_graph, bool lets_in, void (*dependent)(P...), void (*plain)(P...), dim3 grid,
                          unsigned threads, size_t smem, cudaStream_t stream, A... args) {
    const bool captured = stream_captured(stream), overlap = captured ? in_graph && behind_own_kernel(stream) : in_stream;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = overlap ? 1 : 0;
    const cudaError_t err = cudaLaunchKernelEx(&cfg, overlap ? dependent : plain, static_cast<P>(args)...);
    if (captured && lets_in && err == cudaSuccess) note_captured_kernel(stream);
    return err;
}
// Read-only data, in a kernel of either form.
template <bool DEPENDENT, class T>
__device__ __forceinline__ T load_input(const T *p) { return DEPENDENT ? *p : __ldg(p); }
// The next kernel may be launched where there is room for it (its CTAs then wait beside this kernel's).
__device__ __forceinline__ void allow_next_grid() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Everything before this kernel has ended and its results are there.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Launchers implemented one per .cu file; all enqueue on `stream` and return a status.
int launch_validate(const uint8_t *blocks, int64_t groups, int64_t *counts, cudaStream_t stream);
int launch_embedding(const uint8_t *blocks, const int64_t *ids, void *out, bool out_f32,
                     int64_t T, int64_t V, int K, cudaStream_t stream);
int launch_gemv_rows(const uint8_t *blocks, const __half *x, void *y, bool y_f32,
                     int M, int N, int K, cudaStream_t stream);

// Device-side description of an output-row shard whose result is pushed to every rank
// (tq1_linear_f16_sharded): peer pointers are plain device addresses reachable over NVLink.
// Flags are per row tile: word t of a gathered buffer's flag array guards rows [16t, 16t + 16) and is
// stored, with release semantics, by the thread that has just written those rows to that rank.
constexpr int kMaxRanks = 8;
constexpr int kFlagRows = 16;
struct ShardDev {
    int world;                          // <= 1: not sharded, every other field is ignored
    int rank;
    __half *peer_y[kMaxRanks];          // rank p's gathered output, already advanced to this shard's first row
    unsigned *peer_flags[kMaxRanks];    // rank p's tile flags of that output, advanced to this shard's first tile
    const unsigned *epoch_base;         // optional device word added to both epochs (graph replays advance it)
    unsigned publish_epoch;             // value stored to a tile's flag once the tile has been written
    const unsigned *wait_flags;         // local tile flags of the activations this call reads (or null)
    int wait_tiles;                     // how many of them exist
    unsigned wait_epoch;
    int ld_total;                       // row length of the gathered output (elements)
    int swiglu;                         // unsharded only: rows are (gate, up) pairs, y[i] = silu(gate_i) * up_i
};

// Batch-1 GEMV as a persistent chain of links (TMA + integer tensor cores); needs K % 512 == 0, at most
// 128 K chunks and 16-byte aligned blocks. A single product is a chain of one link.
bool gemv_chain_shape_ok(int N, int K);
bool gemv_chain_supported(const uint8_t *blocks, int N, int K);
bool gemv_chain_fits(const uint8_t *blocks, int N, int K);      // also checks the current device's SM count
size_t gemv_chain_workspace_bytes(int N, int K);
size_t gemv_chain_workspace_bound(int N, int K);                // for this matrix and every smaller one
// Two activation rows as exact sums too (more while a sweep is recorded): by the tile kernel, or as M links of one launch over the same
// weights. Launches it (`status` is what came of that) and returns true where one of them takes the call.
bool gemv_looped_shape_ok(int M, int N, int K);
bool try_gemv_looped(const uint8_t *blocks, const __half *x, void *y, bool y_f32, int M, int N, int K, bool swiglu, void *workspace,
                     cudaStream_t stream, int *status);
int gemv_set_loop_tokens(int tokens);       // sweep recording only; process-global
// slot_bytes: room for partial-sum slots behind the workspace's control words
int launch_gemv_single(const uint8_t *blocks, const __half *x, void *y, bool y_f32, int N, int K, bool swiglu,
                       void *workspace, size_t slot_bytes, cudaStream_t stream);
// One or two activation rows with a row's whole sum inside a CTA or a cluster. Launches it (`status` is what came of that; the
// workspace's first word is the status word) and returns true where it takes the call.
bool try_gemv_tiles(const uint8_t *blocks, const __half *x, void *y, bool y_f32, int M, int N, int K, bool swiglu, void *workspace,
                    cudaStream_t stream, int *status);
// How a call is laid out by a kernel that takes it (tests; launches nothing). rooms: null, or how many clusters of 1, 2, .. kMaxCluster CTAs run at once
// (rooms[size]), in place of what the driver says.
struct CallLayout {
    int cluster;                        // CTAs of a cluster
    int sets, stages, tiles;            // sets of warps, ring stages, row tiles of a cluster at most
    bool preferred;                     // over the kernel that takes the call otherwise
};
bool gemv_tiles_layout(int M, int N, int K, const int *rooms, CallLayout *layout);
bool gemm_slices_layout(int M, int N, int K, const int *rooms, CallLayout *layout);
bool gemm_tc_layout(int M, int N, int K, const int *rooms, CallLayout *layout);      // parts of a tile as sets; 1: no cluster adds them up
int launch_shard_wait(const ShardDev &shard, unsigned *status, cudaStream_t stream);
int launch_shard_push(const __half *local, int M, int n_local, const ShardDev &shard, cudaStream_t stream);
int launch_epoch_advance(unsigned *epoch_base, unsigned delta, cudaStream_t stream);

int gemv_noalloc(const uint8_t *blocks, const __half *x, void *y, bool y_f32, int N, int K, cudaStream_t stream);
int gemv_noalloc_status(unsigned *out_host, cudaStream_t stream);

// Batched linear (M >= 2) on tcgen05 tensor cores; needs K % 512 == 0 and 16-byte aligned pointers.
bool gemm_tc_shape_ok(int M, int N, int K);
size_t gemm_tc_workspace_bytes(int M, int N, int K);       // what the call uses
size_t gemm_tc_workspace_bound(int M);                     // what calls of at most M rows use, whatever N and K
int launch_gemm_tc(const uint8_t *blocks, const __half *x, void *y, bool y_f32, int M, int N, int K,
                   void *workspace, cudaStream_t stream, bool swiglu = false);

// silu(gate) * up in FP32, the activation of a gated feed-forward block
__host__ __device__ inline float swiglu_f32(float gate, float up) { return gate / (1.0f + expf(-gate)) * up; }
void gemm_tc_plan(int M, int N, int K, int *tile, int *ctas, int *parts);
int gemm_tc_force_tile(int nt);
bool gemm_tc_forced();
float gemm_tc_few_us(int N, int K);                         // modelled time of a call of up to 16 rows

// Batched linear of 3 to 16 rows on mma.sync; needs K % 512 == 0 and 16-byte aligned pointers.
bool gemm_slices_preferred(int M, int N, int K);            // fits, and faster than the tcgen05 kernel
int launch_gemm_slices(const uint8_t *blocks, const __half *x, void *y, bool y_f32, int M, int N, int K, void *workspace,
                       cudaStream_t stream, bool swiglu = false);
// Launches it (`status` is what came of that) and returns true where it is preferred.
bool try_gemm_slices(const uint8_t *blocks, const __half *x, void *y, bool y_f32, int M, int N, int K, void *workspace,
                     cudaStream_t stream, bool swiglu, int *status);

// Batched linear (M >= 2) with an FP32 sum per group, for every other width and alignment.
bool gemm_groups_preferred(int M, int N, int K);
// The form that takes a call (TQ1_FORM_GROUPS_*); status: the call has a status word, the workspace's first.
int gemm_groups_form(int M, int N, int K, bool status);
int launch_gemm_groups(int form, const uint8_t *blocks, const __half *x, void *y, bool y_f32, int M, int N, int K, unsigned *status,
                       cudaStream_t stream);
float gemm_groups_tc_us(int M, int N, int K);               // modelled time of the tcgen05 form
int launch_gemm_groups_tc(const uint8_t *blocks, const __half *x, void *y, bool y_f32, int M, int N, int K, unsigned *status,
                          cudaStream_t stream);

// Five base-3 digits of a byte packed two bits each (digit i at bits 2i..2i+1).
__host__ __device__ inline uint32_t trits_2bit(uint32_t byte) {
    uint32_t e = 0;
    for (int i = 0; i < 5; ++i) {
        e |= (byte % 3u) << (2 * i);
        byte /= 3u;
    }
    return e;
}

}  // namespace tq1
