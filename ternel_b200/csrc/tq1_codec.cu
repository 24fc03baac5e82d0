// Host-side TQ1_G128 codec and the device-side load-time byte scan.
//
// pack/unpack/validate restate src/bonsai_tq1/format.py:66-122 of the reference;
// tile/untile restate src/bonsai_tq1/lut23_reorder.py:126-165 for row counts the
// tile divides (the MLX layout, src/ternel_mlx/layout.py:76-80).
#include <stdarg.h>
#include <stdio.h>
#include <string.h>
#if defined(__x86_64__)
#include <emmintrin.h>
#endif

#include <algorithm>
#include <atomic>
#include <thread>
#include <vector>

#include "tq1_common.cuh"

#ifdef TQ1_BOUNDS_CHECK
namespace tq1 {
__device__ unsigned long long g_tq1_bounds[4] = {0, 0, 0, 0};
}
#endif

namespace tq1 {

static thread_local char g_error[512] = "";

int fail(int code, const char *fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_error, sizeof(g_error), fmt, ap);
    va_end(ap);
    return code;
}

int cuda_fail(cudaError_t err, const char *what) {
    return fail(TQ1_ERR_CUDA, "%s: %s", what, cudaGetErrorString(err));
}

// f(part, begin, end) over [0, n) in equal contiguous parts, one thread each. A part is at least `grain` items:
// starting a thread costs some 20 us, and a weight of a few hundred KB is done in that time. The threads end with
// the call (nothing is kept between calls, so callers may fork, and may call from several threads at once).
constexpr int kMaxHostThreads = 16;
template <typename F>
static void parallel_parts(int64_t n, int64_t grain, const F &f) {
    const int64_t cores = std::max(1u, std::thread::hardware_concurrency());
    const int parts = (int)std::max<int64_t>(1, std::min<int64_t>({n / grain, cores, kMaxHostThreads}));
    std::thread threads[kMaxHostThreads];
    for (int i = 1; i < parts; ++i) {
        const int64_t begin = n * i / parts, end = n * (i + 1) / parts;
        try {
            threads[i] = std::thread([&f, i, begin, end] { f(i, begin, end); });
        } catch (...) {                             // no thread to be had, or no memory for one: the part runs here
            f(i, begin, end);
        }
    }
    f(0, 0, n / parts);
    for (int i = 1; i < parts; ++i)
        if (threads[i].joinable()) threads[i].join();
}

// check(begin, end) over all of [0, n) in pieces, then, if every one was true, act(begin, end) over the same pieces. Whoever
// has a thread takes the next piece: threads come up 20 us apart, and with equal parts the last one's check kept the
// others waiting (5120x5120 codes: 790 us, this way 540; out of memory instead of cache 740, of which the check is 60). A
// thread with nothing left to check yields until the others are through. Threads started by threads, and threads that act on
// the pieces they have checked, were slower (900).
template <typename C, typename F>
static bool checked_parts(int64_t n, int64_t grain, const C &check, const F &act) {
    const int64_t cores = std::max(1u, std::thread::hardware_concurrency());
    const int workers = (int)std::max<int64_t>(1, std::min<int64_t>({n / grain, cores, kMaxHostThreads}));
    const int64_t piece = workers > 1 ? grain / 4 : std::max<int64_t>(n, 1), pieces = (n + piece - 1) / piece;
    std::atomic<int64_t> to_check{0}, checked{0}, to_act{0};
    std::atomic<bool> good{true};
    const auto work = [&] {
        for (int64_t i; (i = to_check.fetch_add(1)) < pieces; checked.fetch_add(1))
            if (!check(i * piece, std::min(n, (i + 1) * piece))) good.store(false);
        while (checked.load() < pieces) std::this_thread::yield();
        if (!good.load()) return;
        for (int64_t i; (i = to_act.fetch_add(1)) < pieces;) act(i * piece, std::min(n, (i + 1) * piece));
    };
    std::thread threads[kMaxHostThreads];
    for (int i = 1; i < workers; ++i) {
        try {
            threads[i] = std::thread(work);
        } catch (...) {                             // no thread to be had, or no memory for one: the others do its pieces
        }
    }
    work();
    for (std::thread &t : threads)
        if (t.joinable()) t.join();
    return good.load();
}

// Groups per thread of the block codec (28 packed, 128 unpacked bytes each): about 0.1 ms of work.
constexpr int64_t kGroupGrain = 8192;

static void scan_host(const uint8_t *blocks, int64_t groups, int64_t *bad_full, int64_t *bad_tail) {
    int64_t bf[kMaxHostThreads] = {}, bt[kMaxHostThreads] = {};
    parallel_parts(groups, kGroupGrain, [&](int part, int64_t begin, int64_t end) {
        int64_t full = 0, tail = 0;
        for (int64_t g = begin; g < end; ++g) {
            const uint8_t *b = blocks + g * kBlockBytes;
            int over = 0;
            for (int j = 2; j < 27; ++j) over += b[j] > kMaxFull;
            full += over;
            tail += b[27] > kMaxTail;
        }
        bf[part] = full;
        bt[part] = tail;
    });
    *bad_full = *bad_tail = 0;
    for (int i = 0; i < kMaxHostThreads; ++i) { *bad_full += bf[i]; *bad_tail += bt[i]; }
}

// Five codes 0..2 in the low five bytes of w -> c0 + 3 c1 + 9 c2 + 27 c3 + 81 c4. Byte 4 of the product with
// 3^4 + 3^3 2^8 + ... + 3^0 2^32 is that sum; every lower byte's sum is at most 242, so nothing carries into it.
static inline uint8_t pack5(uint64_t w) {
    return (uint8_t)((w * ((81ull) | (27ull << 8) | (9ull << 16) | (3ull << 24) | (1ull << 32))) >> 32);
}
static inline uint64_t load8(const uint8_t *p) {
    uint64_t w;
    memcpy(&w, p, 8);
    return w;
}
// Whether all 128 codes of a group are 0, 1 or 2.
static bool codes_legal(const uint8_t *c) {
    uint64_t over = 0;
    for (int i = 0; i < 16; ++i) {
        const uint64_t w = load8(c + 8 * i);
        over |= (w & 0xfcfcfcfcfcfcfcfcull) | (w & (w >> 1) & 0x0101010101010101ull);      // above 3, or 3
    }
    return over == 0;
}
static void pack_group(const uint8_t *scale, const uint8_t *c, uint8_t *b) {
    b[0] = scale[0];
    b[1] = scale[1];
    for (int j = 0; j < 25; ++j) b[2 + j] = pack5(load8(c + 5 * j));
    b[27] = pack5(load8(c + 120) >> 40);
}

// ---- host arrays to the device -------------------------------------------------------------------------------------
// The driver copies ordinary host memory into pinned memory of its own by the calling thread: 5.7 MB took 313 us, of which the
// transfer is 115. Here the threads of a call fill pieces of the caller's pinned staging, and the calling one enqueues their copies in
// order (a thread's first CUDA call takes longer than a piece: with every thread enqueuing its own 400 us).
//
// The pieces are stored past the caches: the transfer has to ask for lines that are still in a core's cache, and where that core has
// gone idle, as those of a call's threads do, such a transfer took 437 us instead of 125.
static void copy_uncached(unsigned char *dst, const unsigned char *src, size_t n) {      // dst: 16-byte aligned
    size_t i = 0;
#if defined(__x86_64__) && !defined(__CUDA_ARCH__)
    for (; i + 64 <= n; i += 64) {
        const __m128i *from = reinterpret_cast<const __m128i *>(src + i);
        __m128i *to = reinterpret_cast<__m128i *>(dst + i);
        const __m128i a = _mm_loadu_si128(from), b = _mm_loadu_si128(from + 1), c = _mm_loadu_si128(from + 2), e = _mm_loadu_si128(from + 3);
        _mm_stream_si128(to, a);
        _mm_stream_si128(to + 1, b);
        _mm_stream_si128(to + 2, c);
        _mm_stream_si128(to + 3, e);
    }
    memcpy(dst + i, src + i, n - i);
    _mm_sfence();
#else
    memcpy(dst + i, src + i, n - i);
#endif
}
constexpr size_t kUploadPiece = 512 << 10;              // 12 us of transfer (256 KB and 1 MB pieces: 246 and 235 us for 5.7 MB, 213)
constexpr int kUploadThreads = 3;                       // with the calling one as fast as the transfer
struct UploadPart {
    unsigned char *dst;
    const unsigned char *src;
    size_t bytes;
    int64_t pieces;
};

static cudaError_t upload_parts(const UploadPart *parts, unsigned char *staging, size_t piece, int64_t slots, cudaStream_t stream) {
    const int64_t total = parts[0].pieces + parts[1].pieces;
    // Pieces are taken, and enqueued, in order. `filled[i]`: piece i lies in its slot, i % slots; `left`: the pieces before that one
    // have been transferred.
    std::vector<std::atomic<bool>> filled((size_t)total);
    for (std::atomic<bool> &f : filled) f.store(false, std::memory_order_relaxed);
    std::atomic<int64_t> next{0}, left{0};
    const auto place = [&](int64_t i, const UploadPart *&part, size_t &at, size_t &length) {
        part = i < parts[0].pieces ? parts : parts + 1;
        at = (size_t)(i < parts[0].pieces ? i : i - parts[0].pieces) * piece;
        length = std::min(piece, part->bytes - at);
    };
    const auto fill = [&](int64_t i) {
        const UploadPart *part;
        size_t at, length;
        place(i, part, at, length);
        copy_uncached(staging + (size_t)(i % slots) * piece, part->src + at, length);
        filled[i].store(true, std::memory_order_release);
    };
    const auto work = [&] {
        for (int64_t i; (i = next.fetch_add(1)) < total; fill(i))
            while (left.load(std::memory_order_acquire) < i - slots + 1) std::this_thread::yield();
    };
    const int helpers = (int)std::max<int64_t>(0, std::min<int64_t>({total / 4, (int64_t)std::thread::hardware_concurrency() - 1, kUploadThreads}));
    std::thread threads[kUploadThreads];
    for (int i = 0; i < helpers; ++i) {
        try {
            threads[i] = std::thread(work);
        } catch (...) {                                 // no thread to be had, or no memory for one: the others do its pieces
        }
    }
    // half the slots' copies end with an event: who waits for it may fill them again
    const int64_t half = std::max<int64_t>(1, slots / 2);
    cudaEvent_t events[2] = {nullptr, nullptr};
    cudaError_t err = cudaSuccess;
    for (int64_t i = 0; i < total; ++i) {
        if (total > slots && i % half == 0 && i >= 2 * half) {                  // the half before the last one: its transfer is waited for
            const int64_t h = i / half;
            if (err == cudaSuccess) err = cudaEventSynchronize(events[h & 1]);
            left.store((h - 1) * half, std::memory_order_release);
        }
        while (!filled[i].load(std::memory_order_acquire)) {
            // nobody may have taken it; a piece that is not to be filled yet is left alone
            int64_t mine = next.load();
            if (mine < total && left.load() >= mine - slots + 1 && next.compare_exchange_strong(mine, mine + 1)) fill(mine);
            else std::this_thread::yield();
        }
        const UploadPart *part;
        size_t at, length;
        place(i, part, at, length);
        if (err == cudaSuccess)
            err = cudaMemcpyAsync(part->dst + at, staging + (size_t)(i % slots) * piece, length, cudaMemcpyHostToDevice, stream);
        if (total > slots && i % half == half - 1) {
            cudaEvent_t &event = events[(i / half) & 1];
            if (err == cudaSuccess && !event) err = cudaEventCreateWithFlags(&event, cudaEventDisableTiming);
            if (err == cudaSuccess) err = cudaEventRecord(event, stream);
        }
    }
    for (std::thread &t : threads)
        if (t.joinable()) t.join();
    for (cudaEvent_t e : events)
        if (e) cudaEventDestroy(e);
    if (err != cudaSuccess) cudaStreamSynchronize(stream);      // the caller may drop the staging: nothing reads it any more
    return err;
}

// The blocks are scanned as a flat array of 32-bit words, consecutive threads on consecutive words
// (coalesced). Word i of the array is word i % 7 of its block: word 0 holds the scale and two code
// bytes, words 1..5 four code bytes, word 6 three code bytes and the tail byte. Bytes above the limit
// are counted four at a time with a per-byte unsigned compare.
constexpr int kValidateThreads = 224;       // a multiple of 7: a thread always sees the same word of a block
__global__ void __launch_bounds__(kValidateThreads) validate_kernel(const uint32_t *__restrict__ words,
                                                       int64_t groups,
                                                       unsigned long long *__restrict__ counts) {
    unsigned bf = 0, bt = 0;
    const int64_t total = groups * kBlockWords;
    // the grid stride is a multiple of 7 words, so the word's place in its block never changes
    const int pos = threadIdx.x % kBlockWords;
    const uint32_t full_mask = pos == 0 ? 0xffff0000u : pos == 6 ? 0x00ffffffu : 0xffffffffu;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t v = __ldg(words + i);
        // 0xff in every byte that exceeds 242 (as unsigned bytes)
        const uint32_t over = __vcmpgtu4(v, 0xf2f2f2f2u);
        bf += __popc(over & full_mask) >> 3;
        if (pos == 6) bt += (v >> 24) > kMaxTail;
    }
    for (int o = 16; o > 0; o >>= 1) {
        bf += __shfl_xor_sync(0xffffffffu, bf, o);
        bt += __shfl_xor_sync(0xffffffffu, bt, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (bf) atomicAdd(&counts[0], (unsigned long long)bf);
        if (bt) atomicAdd(&counts[1], (unsigned long long)bt);
    }
}

int launch_validate(const uint8_t *blocks, int64_t groups, int64_t *counts, cudaStream_t stream) {
    cudaError_t err = cudaMemsetAsync(counts, 0, 2 * sizeof(int64_t), stream);
    if (err != cudaSuccess) return cuda_fail(err, "tq1_validate_blocks_device: memset");
    if (groups == 0) return TQ1_OK;
    int64_t ctas = (groups * kBlockWords + kValidateThreads - 1) / kValidateThreads;
    if (ctas > 148 * 8) ctas = 148 * 8;
    validate_kernel<<<(unsigned)ctas, kValidateThreads, 0, stream>>>(
        reinterpret_cast<const uint32_t *>(blocks), groups,
        reinterpret_cast<unsigned long long *>(counts));
    err = cudaGetLastError();
    if (err != cudaSuccess) return cuda_fail(err, "tq1_validate_blocks_device: launch");
    return TQ1_OK;
}

// The reference's tiled pair on the device: codes [tiles][gpr][26][tile], scales [tiles][gpr][tile]. A thread takes
// one 28-byte block, consecutive threads consecutive rows of a tile, so a warp reads each code slot as consecutive
// bytes. WRITE = false only counts the bytes above their limit (the load is refused before anything is written).
// A weight of 5120x5120: host scan, relayout and upload 5.9 ms; upload (0.2 ms), these two passes (8 and 12 us) and the read of the
// counts 0.31 ms.
constexpr int kTiledThreads = 128;
template <bool WRITE>
__global__ void __launch_bounds__(kTiledThreads) tiled_kernel(const uint8_t *__restrict__ codes,
                                                              const uint16_t *__restrict__ scales,
                                                              uint32_t *__restrict__ blocks, int64_t rows, int64_t gpr,
                                                              int64_t tile, unsigned long long *counts) {
    if (WRITE && counts && (counts[0] | counts[1])) return;        // the load is refused
    const int64_t r = (int64_t)blockIdx.x * kTiledThreads + threadIdx.x;
    unsigned bf = 0, bt = 0;
    if (r < rows) {
        const int64_t t = r / tile, in = r - t * tile;
        for (int64_t g = blockIdx.y; g < gpr; g += gridDim.y) {
            const uint8_t *src = codes + (t * gpr + g) * kCodeBytes * tile + in;
            uint32_t b[kCodeBytes];
#pragma unroll
            for (int s = 0; s < kCodeBytes; ++s) b[s] = __ldg(src + s * tile);
            if (WRITE) {
                uint32_t *dst = blocks + (r * gpr + g) * kBlockWords;
                if (!TQ1_IN_BOUNDS((r * gpr + g) * kBlockWords + 6, rows * gpr * kBlockWords, 51u)) continue;
                dst[0] = (uint32_t)scales[(t * gpr + g) * tile + in] | (b[0] << 16) | (b[1] << 24);
#pragma unroll
                for (int w = 1; w < kBlockWords; ++w)
                    dst[w] = b[4 * w - 2] | (b[4 * w - 1] << 8) | (b[4 * w] << 16) | (b[4 * w + 1] << 24);
            } else {
#pragma unroll
                for (int s = 0; s < kFullBytes; ++s) bf += b[s] > kMaxFull;
                bt += b[kFullBytes] > kMaxTail;
            }
        }
    }
    if (!WRITE) {
        bf = __reduce_add_sync(0xffffffffu, bf);
        bt = __reduce_add_sync(0xffffffffu, bt);
        if ((threadIdx.x & 31) == 0) {
            if (bf) atomicAdd(&counts[0], (unsigned long long)bf);
            if (bt) atomicAdd(&counts[1], (unsigned long long)bt);
        }
    }
}

// blocks == null: count the bytes above their limit; else write the canonical blocks, unless there are counts that say no.
int launch_tiled(const uint8_t *codes, const uint16_t *scales, uint8_t *blocks, int64_t rows, int64_t gpr, int64_t tile,
                 int64_t *counts, cudaStream_t stream) {
    const dim3 grid((unsigned)((rows + kTiledThreads - 1) / kTiledThreads), (unsigned)std::min<int64_t>(gpr, 256));
    cudaError_t err = !blocks ? cudaMemsetAsync(counts, 0, 2 * sizeof(int64_t), stream) : cudaSuccess;
    if (err != cudaSuccess) return cuda_fail(err, "tq1 tiled blocks: memset");
    auto *c = reinterpret_cast<unsigned long long *>(counts);
    if (!blocks) tiled_kernel<false><<<grid, kTiledThreads, 0, stream>>>(codes, nullptr, nullptr, rows, gpr, tile, c);
    else tiled_kernel<true><<<grid, kTiledThreads, 0, stream>>>(codes, scales, reinterpret_cast<uint32_t *>(blocks), rows,
                                                                gpr, tile, c);
    err = cudaGetLastError();
    return err == cudaSuccess ? TQ1_OK : cuda_fail(err, "tq1 tiled blocks: launch");
}

}  // namespace tq1

using namespace tq1;

extern "C" {

int tq1_abi_version(void) { return 3; }

#ifdef TQ1_BOUNDS_CHECK
// {violations, code of the first, its index, its limit}; copies the record to host memory and clears it.
int tq1_debug_bounds(unsigned long long *out_host) {
    if (cudaMemcpyFromSymbol(out_host, tq1::g_tq1_bounds, sizeof(unsigned long long) * 4) != cudaSuccess) return TQ1_ERR_CUDA;
    const unsigned long long zero[4] = {0, 0, 0, 0};
    if (cudaMemcpyToSymbol(tq1::g_tq1_bounds, zero, sizeof(zero)) != cudaSuccess) return TQ1_ERR_CUDA;
    return TQ1_OK;
}
#endif

const char *tq1_last_error(void) { return g_error; }

int tq1_pack_blocks(const uint8_t *scales, const uint8_t *trits, uint8_t *blocks,
                    int64_t groups, int64_t *n_bad) {
    if (groups < 0 || (groups > 0 && (!scales || !trits || !blocks)))
        return fail(TQ1_ERR_INVALID, "tq1_pack_blocks: null pointer or negative group count");
    // every code is looked at before the first block is written: a refused call leaves the caller's blocks as they were
    const bool good = checked_parts(
        groups, kGroupGrain,
        [&](int64_t begin, int64_t end) {
            bool all = true;
            for (int64_t g = begin; g < end; ++g) all &= codes_legal(trits + g * kGroup);
            return all;
        },
        [&](int64_t begin, int64_t end) {
            for (int64_t g = begin; g < end; ++g)
                pack_group(scales + 2 * g, trits + g * kGroup, blocks + g * kBlockBytes);
        });
    int64_t bad = 0;
    if (!good)
        for (int64_t i = 0; i < groups * kGroup; ++i) bad += trits[i] > 2;
    if (n_bad) *n_bad = bad;
    if (bad) return fail(TQ1_ERR_FORMAT, "source contains %lld non-ternary code(s)", (long long)bad);
    return TQ1_OK;
}

int tq1_validate_blocks(const uint8_t *blocks, int64_t groups,
                        int64_t *n_bad_full, int64_t *n_bad_tail) {
    if (groups < 0 || (groups > 0 && !blocks))
        return fail(TQ1_ERR_INVALID, "tq1_validate_blocks: null pointer or negative group count");
    int64_t bf = 0, bt = 0;
    scan_host(blocks, groups, &bf, &bt);
    if (n_bad_full) *n_bad_full = bf;
    if (n_bad_tail) *n_bad_tail = bt;
    if (bf || bt)
        return fail(TQ1_ERR_FORMAT, "invalid base-3 bytes: regular=%lld, tail=%lld",
                    (long long)bf, (long long)bt);
    return TQ1_OK;
}

int tq1_unpack_blocks(const uint8_t *blocks, uint8_t *scales, uint8_t *trits,
                      int64_t groups, int validate, int64_t *n_bad_full, int64_t *n_bad_tail) {
    if (groups < 0 || (groups > 0 && (!blocks || !scales || !trits)))
        return fail(TQ1_ERR_INVALID, "tq1_unpack_blocks: null pointer or negative group count");
    if (n_bad_full) *n_bad_full = 0;
    if (n_bad_tail) *n_bad_tail = 0;
    if (validate) {
        int rc = tq1_validate_blocks(blocks, groups, n_bad_full, n_bad_tail);
        if (rc != TQ1_OK) return rc;
    }
    uint8_t table[256][5];
    for (unsigned v = 0; v < 256; ++v) {
        unsigned r = v;
        for (int i = 0; i < 5; ++i) { table[v][i] = (uint8_t)(r % 3); r /= 3; }
    }
    parallel_parts(groups, kGroupGrain, [&](int, int64_t begin, int64_t end) {
        for (int64_t g = begin; g < end; ++g) {
            const uint8_t *b = blocks + g * kBlockBytes;
            uint8_t *c = trits + g * kGroup;
            scales[2 * g] = b[0];
            scales[2 * g + 1] = b[1];
            for (int j = 0; j < kFullBytes; ++j) memcpy(c + 5 * j, table[b[2 + j]], 5);
            memcpy(c + 125, table[b[27]], 3);
        }
    });
    return TQ1_OK;
}

int tq1_dequantize_blocks(const uint8_t *blocks, float *out, int64_t groups) {
    if (groups < 0 || (groups > 0 && (!blocks || !out)))
        return fail(TQ1_ERR_INVALID, "tq1_dequantize_blocks: null pointer or negative group count");
    float sign[256][5];                       // byte -> its five weights as -1, 0, +1
    for (unsigned v = 0; v < 256; ++v) {
        unsigned r = v;
        for (int i = 0; i < 5; ++i) { sign[v][i] = (float)((int)(r % 3) - 1); r /= 3; }
    }
    for (int64_t g = 0; g < groups; ++g) {
        const uint8_t *b = blocks + g * kBlockBytes;
        const float d = __half2float(__ushort_as_half((unsigned short)(b[0] | (b[1] << 8))));
        float *y = out + g * kGroup;
        for (int j = 0; j < kFullBytes; ++j)
            for (int i = 0; i < 5; ++i) y[5 * j + i] = sign[b[2 + j]][i] * d;
        for (int i = 0; i < 3; ++i) y[125 + i] = sign[b[27]][i] * d;
    }
    return TQ1_OK;
}

int tq1_tile_blocks(const uint8_t *blocks, uint8_t *codes, uint16_t *scales,
                    int64_t rows, int64_t gpr, int64_t tile) {
    if (rows <= 0 || gpr <= 0 || tile <= 0 || !blocks || !codes || !scales)
        return fail(TQ1_ERR_INVALID, "tq1_tile_blocks: dimensions must be positive and pointers non-null");
    if (rows % tile)
        return fail(TQ1_ERR_INVALID, "tile %lld does not divide %lld rows", (long long)tile, (long long)rows);
    parallel_parts(rows, kGroupGrain / gpr + 1, [&](int, int64_t begin, int64_t end) {
      for (int64_t r = begin; r < end; ++r) {
        int64_t t = r / tile, in = r % tile;
        for (int64_t g = 0; g < gpr; ++g) {
            const uint8_t *b = blocks + (r * gpr + g) * kBlockBytes;
            scales[(t * gpr + g) * tile + in] = (uint16_t)(b[0] | (b[1] << 8));
            uint8_t *dst = codes + ((t * gpr + g) * kCodeBytes) * tile + in;
            for (int s = 0; s < kCodeBytes; ++s) dst[s * tile] = b[2 + s];
        }
      }
    });
    return TQ1_OK;
}

int tq1_untile_blocks(const uint8_t *codes, const uint16_t *scales, uint8_t *blocks,
                      int64_t rows, int64_t gpr, int64_t tile) {
    if (rows <= 0 || gpr <= 0 || tile <= 0 || !blocks || !codes || !scales)
        return fail(TQ1_ERR_INVALID, "tq1_untile_blocks: dimensions must be positive and pointers non-null");
    if (rows % tile)
        return fail(TQ1_ERR_INVALID, "tile %lld does not divide %lld rows", (long long)tile, (long long)rows);
    parallel_parts(rows, kGroupGrain / gpr + 1, [&](int, int64_t begin, int64_t end) {
      for (int64_t r = begin; r < end; ++r) {
        int64_t t = r / tile, in = r % tile;
        for (int64_t g = 0; g < gpr; ++g) {
            uint8_t *b = blocks + (r * gpr + g) * kBlockBytes;
            uint16_t s = scales[(t * gpr + g) * tile + in];
            b[0] = (uint8_t)(s & 0xff);
            b[1] = (uint8_t)(s >> 8);
            const uint8_t *src = codes + ((t * gpr + g) * kCodeBytes) * tile + in;
            for (int k = 0; k < kCodeBytes; ++k) b[2 + k] = src[k * tile];
        }
      }
    });
    return TQ1_OK;
}

int tq1_validate_blocks_device(const uint8_t *blocks_dev, int64_t groups,
                               int64_t *counts_dev, void *stream) {
    if (groups < 0 || !counts_dev || (groups > 0 && !blocks_dev))
        return fail(TQ1_ERR_INVALID, "tq1_validate_blocks_device: null pointer or negative group count");
    if (reinterpret_cast<uintptr_t>(blocks_dev) & 3)
        return fail(TQ1_ERR_INVALID, "tq1_validate_blocks_device: blocks must be 4-byte aligned");
    return launch_validate(blocks_dev, groups, counts_dev, static_cast<cudaStream_t>(stream));
}

static int tiled_checked(const void *codes, const void *second, int64_t rows, int64_t gpr, int64_t tile, const char *who) {
    if (rows <= 0 || gpr <= 0 || tile <= 0 || !codes || !second)
        return fail(TQ1_ERR_INVALID, "%s: dimensions must be positive and pointers non-null", who);
    if (rows % tile)
        return fail(TQ1_ERR_INVALID, "tile %lld does not divide %lld rows", (long long)tile, (long long)rows);
    if (rows > ((int64_t)1 << 31)) return fail(TQ1_ERR_INVALID, "%s: too many rows", who);
    return TQ1_OK;
}

int tq1_validate_codes_device(const uint8_t *codes_dev, int64_t rows, int64_t gpr, int64_t tile, int64_t *counts_dev,
                              void *stream) {
    const int rc = tiled_checked(codes_dev, counts_dev, rows, gpr, tile, "tq1_validate_codes_device");
    return rc != TQ1_OK ? rc : launch_tiled(codes_dev, nullptr, nullptr, rows, gpr, tile, counts_dev,
                                            static_cast<cudaStream_t>(stream));
}

int tq1_untile_blocks_device(const uint8_t *codes_dev, const uint16_t *scales_dev, uint8_t *blocks_dev, int64_t rows,
                             int64_t gpr, int64_t tile, void *stream) {
    const int rc = tiled_checked(codes_dev, scales_dev, rows, gpr, tile, "tq1_untile_blocks_device");
    if (rc != TQ1_OK) return rc;
    if (!blocks_dev || (reinterpret_cast<uintptr_t>(blocks_dev) & 3))
        return fail(TQ1_ERR_INVALID, "tq1_untile_blocks_device: blocks must be non-null and 4-byte aligned");
    return launch_tiled(codes_dev, scales_dev, blocks_dev, rows, gpr, tile, nullptr, static_cast<cudaStream_t>(stream));
}

int tq1_upload_pair(void *dst0, const void *src0, size_t bytes0, void *dst1, const void *src1, size_t bytes1, void *staging,
                    size_t staging_bytes, void *stream) {
    if ((bytes0 && (!dst0 || !src0)) || (bytes1 && (!dst1 || !src1)) || !staging || (reinterpret_cast<uintptr_t>(staging) & 15) || staging_bytes < 65536)
        return fail(TQ1_ERR_INVALID, "tq1_upload_pair: null pointer, or not 64 KiB of 16-byte aligned staging");
    const size_t piece = std::min(kUploadPiece, staging_bytes / 4 & ~(size_t)63);
    const UploadPart parts[2] = {
        {static_cast<unsigned char *>(dst0), static_cast<const unsigned char *>(src0), bytes0, (int64_t)((bytes0 + piece - 1) / piece)},
        {static_cast<unsigned char *>(dst1), static_cast<const unsigned char *>(src1), bytes1, (int64_t)((bytes1 + piece - 1) / piece)}};
    try {
        const cudaError_t err = upload_parts(parts, static_cast<unsigned char *>(staging), piece, (int64_t)(staging_bytes / piece) & ~1ll,
                                             static_cast<cudaStream_t>(stream));
        return err == cudaSuccess ? TQ1_OK : cuda_fail(err, "tq1_upload_pair");
    } catch (...) {
        return fail(TQ1_ERR_INVALID, "tq1_upload_pair: out of host memory");
    }
}

int tq1_load_tiled_device(const uint8_t *codes_dev, const uint16_t *scales_dev, uint8_t *blocks_dev, int64_t rows,
                          int64_t gpr, int64_t tile, int64_t *counts_dev, void *stream) {
    if (!scales_dev || !blocks_dev || (reinterpret_cast<uintptr_t>(blocks_dev) & 3))
        return fail(TQ1_ERR_INVALID, "tq1_load_tiled_device: scales must be non-null, blocks non-null and 4-byte aligned");
    const int rc = tq1_validate_codes_device(codes_dev, rows, gpr, tile, counts_dev, stream);
    return rc != TQ1_OK ? rc : launch_tiled(codes_dev, scales_dev, blocks_dev, rows, gpr, tile, counts_dev,
                                            static_cast<cudaStream_t>(stream));
}

}  // extern "C"
