// Batched linear (M >= 2 activation rows) for TQ1_G128 on sm_100a: trits are decoded into FP16 weights in tensor
// memory, activations come to shared memory by TMA, and tcgen05.mma multiplies them into FP32 accumulators in
// tensor memory.
//
// Stands in for the reference's prefill GEMM and small-batch kernels behind packed_matmul
// (src/ternel_mlx/kernels.py:409-858,1287-1357; src/ternel_mlx/modules.py:425-457). As in the reference's GEMM,
// the group scale is folded into the FP16 weight, which is exact: (c-1)*s is -s, 0 or +s
// (src/ternel_mlx/kernels.py:435-440).
//
// An output tile is 128 weight rows x NT activation rows per CTA (with CG = 2 a CTA pair takes 256 weight rows x NT):
//   D[n][m] = sum_k W[n][k] * x[m][k]      (A = W, in tensor memory; B = x tile, K-major FP16, 128-byte swizzle)
// The unit of work is a chunk of a tile: 4 K blocks of 128 columns = 112 packed bytes per row. A segment is a run of
// consecutive chunks of one tile; a CTA (pair) walks the segments it was dealt.
//   decode warps (G groups of four)  A group takes every G-th chunk of a segment. Its warp q fetches the packed bytes
//        of rows 32q..32q+31 of the chunk into a buffer of its own by TMA, so decoding needs no barrier between warps
//        before the operand is complete. Thread = weight row: code byte -> 8-byte table entry of PRMT selectors ->
//        pairs of FP16 weights picked out of [0, s_lo, s_hi, s_hi ^ 0x80] -> 32 registers = 64 K columns, stored to the
//        row's lane of tensor memory.
//        All groups also read out finished accumulators and store the results.
//   one warp   issues tcgen05.mma for the halves (64 K columns) in a fixed order: chunk wave, K block, group, half; the K
//        blocks take turns on one, two or four accumulators, which are added when the segment is read out
//   one warp   fetches the activation tiles in the same order
// Shared memory traffic of the table bounds the decode (two 128-byte wavefronts per 32 code bytes), so decode warps are
// many and keep no state between chunks. Weights are decoded in natural column order (a byte's five trits straddle
// register pairs differently in even and odd bytes, which the wide table holds as two entries), so activations are used
// as they are: an earlier version permuted them in a launch of its own, a tenth of a prefill call.
//
// Segments that cover only a part of a tile's K range leave an FP32 partial tile in the workspace; the CTA that finishes
// the tile's last part (a counter per tile) adds the parts in ascending K order, so results never depend on timing, and no
// CTA waits for another. A separate launch for these sums cost 3 to 14 us. Equal parts of fewer tiles than slots add up in
// clusters (CLUSTERED, below).
//
// Precision: the tensor core adds to an accumulator by truncation, so the error grows with the columns that one accumulator
// covers: 6.3e-7 of the result (2-norm) for 512, 1.2e-6 for 1024, 3.0e-6 for 2560. All of the accumulator area is therefore
// used, by up to four accumulators that share the columns, and shares of tiles are spread so that few tiles stay in one piece.
#include <cuda.h>
#include <math.h>

#include <type_traits>

#include "tq1_async.cuh"

namespace tq1 {

namespace {

constexpr int kTileW = 128;                                         // weight rows per CTA and tile
constexpr int kChunkGroups = 4;
constexpr int kChunkBytes = kChunkGroups * kBlockBytes;             // 112 packed bytes per row
constexpr int kPackBytes = 32 * kChunkBytes;                        // a warp's rows of a chunk: 3584
constexpr int kStageCols = 64;                                      // tensor-memory columns of a K block of FP16 weights

// Variants:
//   S  up to 32 tokens: two CTAs per SM with two decode groups each hide each other's latencies; the narrow table
//      (one 8-byte entry per byte and lane pair, 32 KB) leaves room for that
//   L  33..128 tokens: one CTA per SM, four groups, wide table (even and odd entries, 64 KB)
//   P  larger: CTA pairs (cta_group::2), each CTA holds half of the activation tile, which halves the activation
//      traffic out of L2 and through shared memory
template <int CG_, int G_, bool WIDE_, int PACK_STAGES_, int RING_, int MAX_COLS_, int ACC_COLS_>
struct Variant {
    static constexpr int CG = CG_, G = G_, PACK_STAGES = PACK_STAGES_;
    static constexpr bool WIDE = WIDE_;
    static constexpr int RING = RING_;                              // K blocks of decoded weights in tensor memory
    static constexpr int MAX_COLS = MAX_COLS_;                      // tokens of a tile at most
    static constexpr int ACC_COLS = ACC_COLS_;                      // columns of tensor memory for accumulators
    static constexpr int kDecodeWarps = 4 * G;
    static constexpr int kThreads = 32 * (kDecodeWarps + 2);
    static constexpr int kGroupCols = MAX_COLS / G < 16 ? 16 : MAX_COLS / G;      // columns a group reads out
    static constexpr int kABase = ACC_COLS;
    static constexpr int kTmemCols = G == 2 ? 256 : 512;
    static_assert(kABase + RING * kStageCols <= kTmemCols, "tensor memory budget");
    static constexpr int kMinCtas = G == 2 ? 2 : 1;
    // P reads a segment's results out after the first K block of the next one is decoded. S and L read them out at once: their
    // pace is the decode's, which loses by the interruption (16 tokens of 17408x5120 18.1 us, 19.9 otherwise; 48 of 5120x17408
    // 21.4 and 21.9; only the most tiles gain, 128 of 34816x5120 45.2 and 44.2).
    static constexpr bool kDecodeAhead = CG == 2;
    static constexpr uint32_t kTableBytes = WIDE ? 65536 : 32768;
    // shared-memory window addresses; the wide table sits at a 64 KiB multiple so that one PRMT builds an entry address
    static constexpr uint32_t kBase = 1024;
    static constexpr uint32_t kPackAddr = kBase;
    static constexpr uint32_t kPackOne = kDecodeWarps * kPackBytes;
    static constexpr uint32_t kTableAddr = WIDE ? 65536 : kPackAddr + PACK_STAGES * kPackOne;
    static constexpr uint32_t kBarAddr = WIDE ? kPackAddr + kPackOne : kTableAddr + kTableBytes;
    static constexpr uint32_t kPack2Addr = kTableAddr + kTableBytes;              // wide: second packed stage
    static constexpr uint32_t kBarBytes = 1024;
    static constexpr uint32_t kBAddr = WIDE ? kPack2Addr + (PACK_STAGES - 1) * kPackOne : kBarAddr + kBarBytes;
    static_assert(!WIDE || kBarAddr + kBarBytes <= kTableAddr, "barriers must end below the table");
    static_assert(kBAddr % 1024 == 0, "swizzled tiles start on 1024-byte boundaries");
    static constexpr uint32_t kWindowEnd = G == 2 ? 1024 + 115712 : 233472;
    static constexpr uint32_t kBRoom = kWindowEnd - kBAddr;
    static constexpr uint32_t kSmemBytes = kWindowEnd - kBase;
    __device__ static __forceinline__ uint32_t pack_addr(int warp, int stage) {
        if (WIDE) return (stage == 0 ? kPackAddr : kPack2Addr) + warp * kPackBytes;
        return kPackAddr + stage * kPackOne + warp * kPackBytes;
    }
};
using VariantS = Variant<1, 2, false, 2, 3, 32, 64>;
using VariantL = Variant<1, 4, true, 1, 4, 128, 256>;
using VariantP = Variant<2, 4, true, 1, 4, 256, 256>;

// Table entries. An 8-bit selector picks the two bytes of one FP16 weight out of the pool [0x00, s_lo, s_hi, s_hi ^ 0x80]:
// code 0 -> -s = (1,3), code 1 -> 0 = (0,0), code 2 -> +s = (1,2). A 16-bit selector of two trits is a PRMT control word.
//   even byte (its first trit in the lower half of a register): word0 = (t0,t1) | t4 << 16, word1 = (t2,t3)
//   odd byte: word0 = (t1,t2) | t0 << 16, word1 = (t3,t4)
// The narrow table holds the even form only; an odd byte's pairs then cost two more byte permutes.
// Sixteen copies of an entry (lanes l and l + 16 share one: a 64-bit shared load serves half a warp at a time) make every
// lookup free of bank conflicts. 256 entries (the 13 past 242 decode to zero weights): a byte that escaped the load-time
// scan still reads inside the table.
struct WideTable { uint32_t w[256 * 64]; };
struct NarrowTable { uint32_t w[256 * 32]; };
constexpr uint32_t sel8(uint32_t c) { return c == 0 ? 0x31u : c == 1 ? 0x00u : 0x21u; }
constexpr void digits(int v, uint32_t (&c)[5]) {
    for (int d = 0; d < 5; ++d) { c[d] = sel8((uint32_t)(v % 3)); v /= 3; }
}
constexpr WideTable make_wide() {
    WideTable t{};
    for (int v = 0; v < 243; ++v) {
        uint32_t c[5] = {};
        digits(v, c);
        for (int l = 0; l < 16; ++l) {
            t.w[v * 64 + 2 * l] = c[0] | (c[1] << 8) | (c[4] << 16);
            t.w[v * 64 + 2 * l + 1] = c[2] | (c[3] << 8);
            t.w[v * 64 + 32 + 2 * l] = c[1] | (c[2] << 8) | (c[0] << 16);
            t.w[v * 64 + 32 + 2 * l + 1] = c[3] | (c[4] << 8);
        }
    }
    return t;
}
constexpr NarrowTable make_narrow() {
    NarrowTable t{};
    for (int v = 0; v < 243; ++v) {
        uint32_t c[5] = {};
        digits(v, c);
        for (int l = 0; l < 16; ++l) {
            t.w[v * 32 + 2 * l] = c[0] | (c[1] << 8) | (c[4] << 16);
            t.w[v * 32 + 2 * l + 1] = c[2] | (c[3] << 8);
        }
    }
    return t;
}
__device__ __align__(128) const WideTable g_wide = make_wide();
__device__ __align__(128) const NarrowTable g_narrow = make_narrow();

// Address, in the cluster's shared window, of `addr` in the leading CTA of the pair.
__device__ __forceinline__ uint32_t leader_addr(uint32_t addr) {
    uint32_t d;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(d) : "r"(addr));
    return d;
}
template <int CG>
__device__ __forceinline__ void mbar_arrive_leader(uint32_t bar) {       // bar: from leader_addr() with CG = 2
    // CTA-scope release: what the leader's MMA reads lies in tensor memory and is ordered by tcgen05.wait::st and the
    // tcgen05 fences; a cluster-scope release waits for every global store of the thread (2000 clocks a time)
    if (CG == 2) asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
    else asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Bounded wait: after the limit *status is set and `dead` stops every further wait of the thread, so that the
// kernel ends (with results that the status marks as bad) instead of hanging. The loop is a few instructions: up to
// twenty warps of an SM wait at a time, and what they issue while they do is taken from the decoding ones.
__device__ __forceinline__ void mbar_wait(uint32_t bar, uint32_t parity, unsigned *status, bool &dead) {
    if (dead) return;
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p, q;\n\t.reg .u32 n;\n\t"
                 "mov.u32 n, %3;\n"
                 "TRY:\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 4000;\n\t"
                 "@p bra DONE;\n\t"
                 "sub.u32 n, n, 1;\n\t"
                 "setp.ne.u32 q, n, 0;\n\t"
                 "@q bra TRY;\n"
                 "DONE:\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity), "n"(kSpinLimit) : "memory");
    if (!ok) {
        atomicExch(status, 3u);
        dead = true;
    }
}
// Activation tile half: {64 columns, box rows} at (x, y). With a CTA pair the bytes count on the leader's barrier.
template <int CG>
__device__ __forceinline__ void tma_load_x(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    if (CG == 2)
        asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
                     "[%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
    else
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes "
                     "[%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
// Called by all 32 lanes: one elected lane arms the warp's barrier and requests its 32 rows x 112 bytes.
__device__ __forceinline__ void elected_load_packed(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "elect.sync _|p, 0xffffffff;\n\t"
                 "@p mbarrier.arrive.expect_tx.shared::cta.b64 _, [%4], %5;\n\t"
                 "@p cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n\t}"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar), "n"(kPackBytes) : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
// A operand in tensor memory (lane = weight row, 8 columns per K = 16 step), B in shared memory.
template <int CG>
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                            uint32_t accumulate) {
    if (CG == 2)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                     ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                     ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
// Arrives on `bar` (of both CTAs of a pair) when every MMA issued so far has finished.
template <int CG>
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    if (CG == 2)
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                     ::"r"(bar), "h"((uint16_t)3) : "memory");
    else
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_load16(uint32_t taddr, float *v) {
    uint32_t u[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]),
          "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
        : "r"(taddr) : "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(u[i]);
}

// n / d for 0 <= n < 2^31 by one multiplication: mul = ceil(2^64 / d), so the error n * (mul * d - 2^64) stays below 2^64.
struct Divisor {
    unsigned long long mul;
    int d;
    __host__ __device__ __forceinline__ void set(int divisor) {
        d = divisor;
        mul = divisor > 1 ? ~0ull / (unsigned)divisor + 1 : 0ull;
    }
    __host__ __device__ __forceinline__ int div(int n) const {
        if (d == 1) return n;
#ifdef __CUDA_ARCH__
        return (int)__umul64hi((unsigned long long)(unsigned)n, mul);
#else
        return n / d;
#endif
    }
};

// How the chunks of all tiles, numbered tile-major, are dealt out. A slot is a CTA (a CTA pair with CG = 2).
//   splits > 0: every tile in `splits` equal parts, one part per slot (fewer tiles than slots).
//   splits == 0: every slot first computes whole_rounds whole tiles (slot * whole_rounds + k); the tiles from whole_tiles
//     on are cut into equal contiguous ranges of chunks, one per slot (stream-K), so that all slots do the same number.
struct WorkSplit {
    int total_iters, slots, chunks, splits;
    int quot, rem;                              // total_iters = slots * quot + rem: `rem` ranges get one more
    int spread;                                 // those lie between the others, else they come first
    int whole_rounds, whole_tiles;
    int tiles_total;                            // output tiles of the call (a slot's last whole tiles may lie beyond)
    Divisor by_splits, by_chunks, by_slots;
    __host__ __device__ __forceinline__ int first_iter(int slot) const {
        if (slot >= slots) return total_iters;
        if (splits == 0) return spread ? by_slots.div(slot * total_iters) : slot * quot + (slot < rem ? slot : rem);
        const int tile = by_splits.div(slot), part = slot - tile * splits;
        return tile * chunks + by_splits.div(chunks * part);
    }
};

// A slot's segments in order: its whole tiles, then the pieces of its range of the shared tiles.
struct SegmentWalk {
    const WorkSplit &work;                      // kernel parameters: read where they are used, not kept in registers
    int slot, round, it, pieces;
    __device__ __forceinline__ SegmentWalk(const WorkSplit &work_, int slot_)
        : work(work_), slot(slot_), round(0), it(work_.first_iter(slot_)), pieces(0) {}
    // end: work.first_iter(slot + 1); part: which of the slot's two partial-tile areas a partial segment is stored to
    __device__ __forceinline__ bool next(int end, int &tile, int &c0, int &len, int &part) {
        if (round < work.whole_rounds && slot * work.whole_rounds + round < work.tiles_total) {
            tile = slot * work.whole_rounds + round++;
            c0 = 0;
            len = work.chunks;
            part = 0;
            return true;
        }
        if (it >= end) return false;
        const int t = work.by_chunks.div(it);
        c0 = it - t * work.chunks;
        len = min(work.chunks - c0, end - it);
        tile = work.whole_tiles + t;
        part = pieces++ == 0 ? 0 : 1;
        it += len;
        return true;
    }
};

// The one segment of a slot where every tile is cut into equal parts (splits > 0).
struct OneSegment {
    const WorkSplit &work;
    int slot;
    bool taken;
    __device__ __forceinline__ OneSegment(const WorkSplit &work_, int slot_) : work(work_), slot(slot_), taken(false) {}
    __device__ __forceinline__ bool next(int end, int &tile, int &c0, int &len, int &part) {
        if (taken) return false;
        taken = true;
        tile = work.by_splits.div(slot);
        c0 = work.first_iter(slot) - tile * work.chunks;
        len = end - work.first_iter(slot);
        part = 0;
        return true;
    }
};

struct GemmParams {
    void *y;                  // [M][N] (FP16/FP32), with swiglu [M][N / 2]
    float *partials;          // [2 * CTAs][nt][128] FP32
    unsigned *counters;       // per shared tile (and CTA of a pair): parts stored so far; zero between calls
    unsigned *status;
    int M, N, groups;         // groups: K / 128
    int tiles_m;              // token tiles; output tile t covers weight tile t / tiles_m, token tile t % tiles_m
    Divisor by_tiles_m;
    int nt;                   // tokens per tile, a multiple of 16 * CG; the last token tile takes what is left
    int accs, acc_cols;       // accumulators (1, 2 or 4) and the columns from one to the next
    int b_stages, b_rows;     // activation ring: stages and rows per CTA of one stage
    WorkSplit work;
    int y_f32;
    int pair_y, quad_y;       // results of two (FP16) or four neighbouring rows may be stored at a time
};

// GATED: the rows are (gate, up) pairs. A kernel of its own: the gates' code in the common one cost 3% of long prompts (777 tokens
// of 34816x5120 without gates 204 us, 199 apart) and 7% of the shortest calls (17 of 1000x1024 5.8 us, 5.4).
// CLUSTERED: every tile is cut into equal parts, and the CTAs of a cluster, one for each, add them through distributed shared
// memory. Through the workspace a part's way out, the count and the sum by the last CTA took 4 us of a call. The same build with the
// parts in the workspace and in a cluster, calls in a row (us): 20 tokens of 4096x4096 8.4 and 7.4, 100 of 1024x5120 9.4 and 7.9, 129 of
// 66x5120 8.7 and 6.9, 100 of 130x12288 12.0 and 8.0, 48 of 5120x17408 19.8 and 19.9. Beside another stream's kernels a cluster waits
// until a GPC has room for all of it: with 4096^3 products of bf16 there the five calls take 38 and 55, 26 and 40, 10 and 11, 18 and 39,
// 68 and 70 us. A kernel of its own too: addresses of a CTA in a cluster take a register, for which only the walk over several
// segments makes room (64 tokens of 17408x5120 as one kernel 21.3 -> 23.4 us).
template <class V, bool GATED, bool CLUSTERED>
__global__ void __launch_bounds__(V::kThreads, V::kMinCtas)
tq1_gemm_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap,
                const __grid_constant__ GemmParams prm) {
    constexpr int CG = V::CG, G = V::G, RING = V::RING, kDecode = V::kDecodeWarps;
    constexpr int kMmaWarp = kDecode, kXWarp = kDecode + 1;
    extern __shared__ __align__(1024) unsigned char smem[];
    // In a cluster launch the upper byte of a shared-memory address names the CTA; the offsets below it are fixed.
    const uint32_t window = (uint32_t)__cvta_generic_to_shared(smem);
    const uint32_t wbase = CG == 2 || CLUSTERED ? window & 0xff000000u : 0u;
    if (window != wbase + V::kBase) {                                // the fixed window addresses do not hold
        if (threadIdx.x == 0) atomicExch(prm.status, 2u);
        return;
    }
    // EMPTY[i % READ_BARS]: the MMAs of K block i have read both operands. A barrier tells one phase from the next only; with
    // four per ring stage a group knows a block that is up to four uses of the stage ahead of the last one it waited for.
    constexpr int READ_BARS = V::kDecodeAhead ? 4 * RING : RING;
    constexpr int TAB = 0, PACK = 1, FULL_A = PACK + kDecode * V::PACK_STAGES, FULL_B = FULL_A + RING,
                  EMPTY = FULL_B + RING, ACC_FULL = EMPTY + READ_BARS, ACC_FREE = ACC_FULL + 1, NUM_BARS = ACC_FREE + 1;
    static_assert(NUM_BARS * 8 <= 1000, "barrier area");
    auto bar = [wbase](int i) { return wbase + V::kBarAddr + 8u * (uint32_t)i; };
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(smem + (V::kBarAddr - V::kBase) + 1008);
    volatile uint32_t *last_flag = tmem_slot + 1;

    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int slot = CG == 2 ? blockIdx.x >> 1 : blockIdx.x, rank = CG == 2 ? blockIdx.x & 1 : 0;

    // ---- set-up that depends on no earlier kernel: barriers, decode table, tensor memory ---------------------
    if (tid == 0) {
        mbar_init(bar(TAB), 1);
        for (int i = 0; i < kDecode * V::PACK_STAGES; ++i) mbar_init(bar(PACK + i), 1);
        for (int i = 0; i < RING; ++i) {
            mbar_init(bar(FULL_A + i), 4 * CG);
            mbar_init(bar(FULL_B + i), 1);
        }
        for (int i = 0; i < READ_BARS; ++i) mbar_init(bar(EMPTY + i), 1);
        mbar_init(bar(ACC_FULL), 1);
        mbar_init(bar(ACC_FREE), kDecode * CG);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_expect_tx(bar(TAB), V::kTableBytes);
        if (V::WIDE) bulk_load(wbase + V::kTableAddr, &g_wide, V::kTableBytes, bar(TAB));
        else bulk_load(wbase + V::kTableAddr, &g_narrow, V::kTableBytes, bar(TAB));
    }
    if (warp == kMmaWarp) {
        const uint32_t where = wbase + V::kBarAddr + 1008;
        if (CG == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(where), "r"((uint32_t)V::kTmemCols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(where), "r"((uint32_t)V::kTmemCols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
        // The next kernel in the stream may start its own set-up from now on: not before this CTA has its tensor memory (a CTA of that
        // kernel beside it could take it, and waits for this kernel), and no later: beside another stream's kernels a launch that
        // comes after what is set up below finds no SM for longer (48 tokens of 5120x17408 beside elementwise kernels 99 us, now 81).
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    // The segments, and for a decode warp the packed bytes that it requests ahead of its decoding: the walks are set up and the
    // first bytes brought to L2 (a hint, whatever they hold by now) while earlier kernels run. Behind the wait below this
    // took 4700 clocks up to the first decoded byte, now 2800.
    auto weight_tile = [&](int t) { return prm.by_tiles_m.div(t); };
    auto token_tile0 = [&](int t) { return (t - prm.by_tiles_m.div(t) * prm.tiles_m) * prm.nt; };     // first token
    // tokens of a token tile, as the MMA's N (whole steps of 16 per CTA)
    auto tile_tokens = [&](int m0) {
        const int left = min(prm.nt, prm.M - m0);
        return (left + 16 * CG - 1) / (16 * CG) * (16 * CG);
    };
    using Walk = std::conditional_t<CLUSTERED, OneSegment, SegmentWalk>;
    Walk walk(prm.work, slot), pwalk(prm.work, slot);
    const int end_iter = prm.work.first_iter(slot + 1);
    int p_tile = 0, p_c0 = 0, p_len = 0, p_part, p_unit = warp >> 2;
    auto seek = [&]() -> bool {
        while (p_unit >= p_len) {
            if (!pwalk.next(end_iter, p_tile, p_c0, p_len, p_part)) { p_len = 0; return false; }
            p_unit = warp >> 2;
        }
        return true;
    };
    auto packed_row = [&]() { return (weight_tile(p_tile) * CG + rank) * kTileW + (warp & 3) * 32; };
    // the results of four neighbouring rows from nq of token m
    auto store_quad = [&](float (&r)[4], int m, int nq) {
        int count = min(4, prm.N - nq);
        size_t o = (size_t)m * prm.N + nq;
        size_t limit = (size_t)prm.M * prm.N;
        if (GATED) {
            r[0] = swiglu_f32(r[0], r[1]);
            r[1] = swiglu_f32(r[2], r[3]);
            count >>= 1;
            o = (size_t)m * (prm.N >> 1) + (nq >> 1);
            limit >>= 1;
        }
        if (CG == 2 && prm.quad_y) {                    // all at once; N is a multiple of four. (For shorter calls the code costs more: +0.2 us.)
            if (count <= 0 || !TQ1_IN_BOUNDS(o + count - 1, limit, 40u)) return;
            const __half2 h0 = __floats2half2_rn(r[0], r[1]), h1 = __floats2half2_rn(r[2], r[3]);
            const uint2 h = make_uint2(reinterpret_cast<const uint32_t &>(h0), reinterpret_cast<const uint32_t &>(h1));
            if (GATED && prm.y_f32) *reinterpret_cast<float2 *>(static_cast<float *>(prm.y) + o) = make_float2(r[0], r[1]);
            else if (GATED) *reinterpret_cast<uint32_t *>(static_cast<__half *>(prm.y) + o) = h.x;
            else if (prm.y_f32) *reinterpret_cast<float4 *>(static_cast<float *>(prm.y) + o) = make_float4(r[0], r[1], r[2], r[3]);
            else *reinterpret_cast<uint2 *>(static_cast<__half *>(prm.y) + o) = h;
            return;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (e < count && TQ1_IN_BOUNDS(o + e, limit, 40u)) {
                if (prm.y_f32) static_cast<float *>(prm.y)[o + e] = r[e];
                else static_cast<__half *>(prm.y)[o + e] = __float2half_rn(r[e]);
            }
        }
    };
    if (warp < kDecode) {
        if (seek() && packed_row() < prm.N && elect_one())          // rows past the end are filled in, not fetched
            asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];"
                         ::"l"(&wmap), "r"((p_c0 + p_unit) * kChunkBytes), "r"(packed_row()) : "memory");
        __syncwarp();
    }
    if (warp == kXWarp && elect_one()) asm volatile("prefetch.tensormap [%0];" ::"l"(&xmap) : "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (CG == 2) {
        asm volatile("barrier.cluster.arrive.release;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    } else {
        __syncthreads();
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    // everything below touches memory that earlier kernels may have written or may still read
    asm volatile("griddepcontrol.wait;" ::: "memory");

    bool dead = false;
    int tile, c0, len, part;


    // K blocks are numbered in the order the MMA warp takes them, over all segments: block i of a CTA uses stage i % RING of
    // the decoded weights and stage i % b_stages (<= RING) of the activations. One commit (EMPTY) says to decoders and
    // activations alike that its MMAs have read both.
    // A wave is the G chunks (fewer at a segment's end) that the groups decode side by side; its blocks are ordered by K
    // block first.
    if (warp == kXWarp) {
        // ------------------------------------------------------------------ activation tiles
        if (elect_one()) {
            uint32_t stage = 0, freed = 0, phase = 0, filled = 0;      // freed: barrier of the block that used this buffer before
            const uint32_t bytes = (uint32_t)prm.b_rows * 256u;
            while (walk.next(end_iter, tile, c0, len, part)) {
                const int m0 = token_tile0(tile);
                const int row = m0 + (CG == 2 ? rank * (tile_tokens(m0) / 2) : 0);
                for (int u0 = 0; u0 < len; u0 += G) {
                    const int width = min(G, len - u0), k0 = (c0 + u0) * kChunkGroups;
                    for (int kb = 0; kb < kChunkGroups; ++kb) {
                        for (int g = 0; g < width; ++g) {
                            const int k = k0 + g * kChunkGroups + kb;
                            if (filled < (uint32_t)prm.b_stages) {
                                ++filled;
                            } else {
                                mbar_wait(bar(EMPTY + freed), phase, prm.status, dead);
                                if (++freed == READ_BARS) { freed = 0; phase ^= 1u; }
                            }
                            if (dead) break;
                            const uint32_t full = CG == 2 ? leader_addr(bar(FULL_B + stage)) : bar(FULL_B + stage);
                            if (rank == 0) mbar_expect_tx(bar(FULL_B + stage), CG * bytes);
                            const uint32_t dst = wbase + V::kBAddr + stage * bytes;
                            tma_load_x<CG>(dst, &xmap, k * kGroup, row, full);
                            tma_load_x<CG>(dst + bytes / 2, &xmap, k * kGroup + 64, row, full);
                            if (++stage == (uint32_t)prm.b_stages) stage = 0;
                        }
                    }
                }
            }
        }
    } else if (warp == kMmaWarp) {
        // ------------------------------------------------------------------ MMA issue (leading CTA of a pair)
        if (rank == 0 && elect_one()) {
            uint32_t bstage = 0, bphase = 0, astage = 0, aphase = 0, read = 0, seg = 0;
            const uint32_t b_bytes = (uint32_t)prm.b_rows * 256u;
            while (walk.next(end_iter, tile, c0, len, part)) {
                const int n_tok = tile_tokens(token_tile0(tile));
                // FP32 accumulate, FP16 A and B, both K-major, M = 128 per CTA, N = tokens
                const uint32_t idesc = (1u << 4) | ((uint32_t)(n_tok >> 3) << 17) | ((uint32_t)(kTileW * CG >> 4) << 24);
                const int blocks = len * kChunkGroups;
                if (seg > 0) mbar_wait(bar(ACC_FREE), (seg - 1) & 1u, prm.status, dead);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int i = 0; i < blocks; ++i) {
                    mbar_wait(bar(FULL_B + bstage), bphase, prm.status, dead);
                    mbar_wait(bar(FULL_A + astage), aphase, prm.status, dead);
                    if (dead) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t a_tmem = tmem_base + (uint32_t)V::kABase + astage * kStageCols;
                    const uint32_t b_addr = wbase + V::kBAddr + bstage * b_bytes;
                    const uint64_t b_lo = umma_desc(b_addr), b_hi = umma_desc(b_addr + b_bytes / 2);
                    const uint32_t acc = tmem_base + (uint32_t)((i & (prm.accs - 1)) * prm.acc_cols);
#pragma unroll
                    for (int j = 0; j < 8; ++j)                    // K = 16 steps: four of each 64-wide swizzle atom
                        umma_f16_ts<CG>(acc, a_tmem + 8u * j, (j < 4 ? b_lo : b_hi) + 2u * (j & 3), idesc,
                                        (i >= prm.accs || j > 0) ? 1u : 0u);
                    umma_commit<CG>(bar(EMPTY + read));
                    if (++read == READ_BARS) read = 0;
                    if (++astage == RING) { astage = 0; aphase ^= 1u; }
                    if (++bstage == (uint32_t)prm.b_stages) { bstage = 0; bphase ^= 1u; }
                }
                if (!dead) umma_commit<CG>(bar(ACC_FULL));
                ++seg;
            }
        }
    } else {
        // ------------------------------------------------------------------ decode and results
        const int group = warp >> 2, quad = warp & 3;
        const int row_in_tile = quad * 32 + lane;                       // = tensor-memory lane
        const uint32_t tmem_lane = tmem_base + ((uint32_t)(quad * 32) << 16);
        const uint32_t lane_entry = wbase + V::kTableAddr + (uint32_t)(lane & 15) * 8u;

        uint32_t requested = 0, consumed = 0;
        auto request = [&]() {
            if (!seek()) return;
            const uint32_t s = requested % V::PACK_STAGES;
            elected_load_packed(wbase + V::pack_addr(warp, (int)s), &wmap, (p_c0 + p_unit) * kChunkBytes, packed_row(),
                                bar(PACK + warp * V::PACK_STAGES + (int)s));
            ++requested;
            p_unit += G;
        };
#pragma unroll
        for (int s = 0; s < V::PACK_STAGES; ++s) request();

        int block0 = 0;                                                 // number of the wave's first K block
        int seen = -1;                                                  // the newest K block waited for: its MMAs have read it
        auto wait_read = [&](int block) {
            if (block < 0) return;
            seen = block;
            mbar_wait(bar(EMPTY + block % READ_BARS), (uint32_t)(block / READ_BARS) & 1u, prm.status, dead);
        };
        uint32_t seg = 0;
        mbar_wait(bar(TAB), 0, prm.status, dead);

        // Reads out a segment's accumulators and stores its results.
        auto finish = [&](int tile, int len, int part) {
            const int m0 = token_tile0(tile), n_tok = tile_tokens(m0);
            const int n = (weight_tile(tile) * CG + rank) * kTileW + row_in_tile;
            const int per_group = (n_tok / 16 + G - 1) / G * 16;
            const int c_begin = group * per_group, cols = min(per_group, n_tok - c_begin);     // cols <= 0: none
            const bool whole = !CLUSTERED && len == prm.work.chunks;
            // the slots that share this tile, worked out while the last products are still being added
            const int shared_tile = tile - prm.work.whole_tiles, it0 = shared_tile * prm.work.chunks;
            int lo = slot, hi = slot;
            if (CLUSTERED) {
            } else if (!whole && prm.work.splits > 0) {
                lo = shared_tile * prm.work.splits;
                hi = lo + prm.work.splits - 1;
            } else if (!whole) {
                while (prm.work.first_iter(lo) > it0) --lo;
                while (prm.work.first_iter(hi + 1) < it0 + prm.work.chunks) ++hi;
            }
            mbar_wait(bar(ACC_FULL), seg & 1u, prm.status, dead);
            ++seg;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            constexpr int kStep = 16;                                                          // columns in registers at a time
            auto read_step = [&](int s0, float (&v)[kStep]) {
#pragma unroll
                for (int c = 0; c < kStep; ++c) v[c] = 0.0f;
                for (int a = 0; a < prm.accs && s0 < cols; ++a) {
                    float u[kStep];
                    tmem_load16(tmem_lane + (uint32_t)(a * prm.acc_cols + c_begin + s0), u);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int c = 0; c < kStep; ++c) {
                        asm volatile("" : "+f"(u[c]));                                         // no use before the wait
                        v[c] += u[c];
                    }
                }
            };
            auto release = [&]() {                      // the next segment may overwrite the accumulators
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive_leader<CG>(CG == 2 ? leader_addr(bar(ACC_FREE)) : bar(ACC_FREE));
            };
            const int tokens = min(cols, prm.M - (m0 + c_begin));                              // of the group's columns
            const int out_n = GATED ? prm.N >> 1 : prm.N;
            if (CLUSTERED) {             // a part of the tile's K range: kept as FP32 where the activations were
#pragma unroll 1
                for (int s0 = 0; s0 < V::kGroupCols; s0 += kStep) {
                    float v[kStep];
                    read_step(s0, v);
                    float *to = reinterpret_cast<float *>(smem + (V::kBAddr - V::kBase)) + (c_begin + s0) * kTileW + row_in_tile;
#pragma unroll
                    for (int c = 0; c < kStep; ++c)
                        if (s0 + c < tokens) to[c * kTileW] = v[c];
                }
                return;
            }
            if (!whole) {                               // a part of the tile's K range: kept as FP32
                const size_t area = (size_t)prm.nt * kTileW;
                float *slot_part = prm.partials + ((size_t)2 * blockIdx.x + part) * area + row_in_tile;
#pragma unroll 1
                for (int s0 = 0; s0 < V::kGroupCols; s0 += kStep) {
                    float v[kStep];
                    read_step(s0, v);
                    if (s0 + kStep >= V::kGroupCols) release();
                    const int col0 = c_begin + s0;
#pragma unroll
                    for (int c = 0; c < kStep; ++c)
                        if (s0 + c < tokens && TQ1_IN_BOUNDS((size_t)(col0 + c) * kTileW + row_in_tile, area, 41u))
                            __stcg(slot_part + (size_t)(col0 + c) * kTileW, v[c]);
                }
                // The slot that completes the tile's count adds the parts.
                asm volatile("bar.sync 1, %0;" ::"n"(kDecode * 32) : "memory");
                if (tid == 0) {
                    // the barrier orders the other warps' stores before this thread's release, and its acquire before their reads
                    unsigned *counter = prm.counters + shared_tile * CG + rank, before;
                    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(before) : "l"(counter) : "memory");
                    const bool last = before == (unsigned)(hi - lo);
                    if (last) *counter = 0u;                // zero for the next call
                    if (before > (unsigned)(hi - lo)) atomicExch(prm.status, 8u);     // it was not zero when the call began
                    *last_flag = last ? 1u : 0u;
                }
                asm volatile("bar.sync 1, %0;" ::"n"(kDecode * 32) : "memory");
                if (*last_flag == 0u) return;
                const int all = min(n_tok, prm.M - m0), quads = all * (kTileW / 4);      // four rows of a column each
                constexpr int kThreadsR = kDecode * 32, kFlight = 4;
                const int tile_n0 = (weight_tile(tile) * CG + rank) * kTileW;
                for (int i0 = tid; i0 < quads; i0 += kThreadsR * kFlight) {
                    float4 total[kFlight];
#pragma unroll
                    for (int f = 0; f < kFlight; ++f) total[f] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 2
                    for (int sl = lo; sl <= hi; ++sl) {
                        // the tile is that slot's first segment of shared tiles if its range starts inside the tile
                        const int which = prm.work.splits > 0 || prm.work.first_iter(sl) >= it0 ? 0 : 1;
                        const float4 *src = reinterpret_cast<const float4 *>(
                            prm.partials + ((size_t)2 * (sl * CG + rank) + which) * area);
#pragma unroll
                        for (int f = 0; f < kFlight; ++f) {
                            const int i = i0 + f * kThreadsR;
                            const float4 p = i < quads ? __ldcg(src + i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                            total[f].x += p.x; total[f].y += p.y; total[f].z += p.z; total[f].w += p.w;
                        }
                    }
#pragma unroll
                    for (int f = 0; f < kFlight; ++f) {
                        const int i = i0 + f * kThreadsR, m = m0 + (i >> 5), nq = tile_n0 + (i & 31) * 4;
                        if (i >= quads) break;
                        float r[4] = {total[f].x, total[f].y, total[f].z, total[f].w};
                        store_quad(r, m, nq);
                    }
                }
                return;
            }
            if (GATED || (!prm.y_f32 && prm.pair_y)) {
                // Neighbouring rows are neighbouring results, and neighbouring lanes. Two lanes exchange columns, so that the even
                // one has both rows of column c and the odd one of column c + 1: half as many stores, and with gate and up rows
                // every lane has a result to work out. Results wait in registers until the accumulators are given back; gate and
                // up themselves, twice as many, spill (777 tokens of 34816x5120 without gates 203 -> 216 us, as one kernel).
                const int odd = lane & 1, row = n - odd;
                uint32_t held[V::kGroupCols / 2];
#pragma unroll
                for (int s0 = 0; s0 < V::kGroupCols; s0 += kStep) {
                    float v[kStep];
                    read_step(s0, v);
#pragma unroll
                    for (int c = 0; c < kStep; c += 2) {
                        const float other = __shfl_xor_sync(0xffffffffu, odd ? v[c] : v[c + 1], 1);
                        const float first = odd ? other : v[c], second = odd ? v[c + 1] : other;
                        uint32_t &result = held[(s0 + c) / 2];
                        if (GATED) {
                            const float out = swiglu_f32(first, second);
                            result = prm.y_f32 ? __float_as_uint(out) : (uint32_t)__half_as_ushort(__float2half_rn(out));
                        } else {
                            const __half2 out = __floats2half2_rn(first, second);
                            result = reinterpret_cast<const uint32_t &>(out);
                        }
                    }
                }
                release();
                size_t o = (size_t)(m0 + c_begin + odd) * out_n + (GATED ? row >> 1 : row);
                const bool in_rows = row + 1 < prm.N;                  // N is even here
#pragma unroll
                for (int c = 0; c < V::kGroupCols; c += 2) {
                    if (c + odd < tokens && in_rows && TQ1_IN_BOUNDS(o + (GATED ? 0 : 1), (size_t)prm.M * out_n, 40u)) {
                        if (!GATED) *reinterpret_cast<uint32_t *>(static_cast<__half *>(prm.y) + o) = held[c / 2];
                        else if (prm.y_f32) static_cast<float *>(prm.y)[o] = __uint_as_float(held[c / 2]);
                        else static_cast<__half *>(prm.y)[o] = __ushort_as_half((unsigned short)held[c / 2]);
                    }
                    o += 2 * (size_t)out_n;
                }
                return;
            }
            if constexpr (!GATED) {
#pragma unroll 1
                for (int s0 = 0; s0 < V::kGroupCols; s0 += kStep) {
                    float v[kStep];
                    read_step(s0, v);
                    if (s0 + kStep >= V::kGroupCols) release();
                    const size_t o = (size_t)(m0 + c_begin + s0) * prm.N + n;
#pragma unroll
                    for (int c = 0; c < kStep; ++c) {
                        if (n < prm.N && s0 + c < tokens && TQ1_IN_BOUNDS(o + (size_t)c * prm.N, (size_t)prm.M * prm.N, 40u)) {
                            if (prm.y_f32) static_cast<float *>(prm.y)[o + (size_t)c * prm.N] = v[c];
                            else static_cast<__half *>(prm.y)[o + (size_t)c * prm.N] = __float2half_rn(v[c]);
                        }
                    }
                }
            }
        };

        // A segment's results are read out when the group has decoded its first K block of the next one: the ring is full
        // again by then, and the MMAs go on as soon as the accumulators are in registers, over the stores too (2048 tokens of
        // 17408x5120 253 us with the results first, 240 now; 777 of 34816x5120 213 and 199, with gates 251 and 219).
        int done_tile = 0, done_len = 0, done_part = 0;                 // the segment that waits for it (length 0: none)
        for (;;) {
            const bool more = walk.next(end_iter, tile, c0, len, part);
            if (!more) len = V::kDecodeAhead ? 1 : 0;                   // one more turn, for the last segment's results
            for (int u0 = 0; u0 < len; u0 += G) {
                const int width = min(G, len - u0), unit = u0 + group;
                const int wave0 = block0;
                block0 += width * kChunkGroups;
                const bool active = more && unit < len;
                // This row's 112 bytes come into registers in three steps (all at once spills); after the last the buffer is
                // free for the next request.
                uint32_t words[4 * 7];
                const uint32_t s = consumed % V::PACK_STAGES;
                const uint32_t src = wbase + V::pack_addr(warp, (int)s) + (uint32_t)lane * kChunkBytes;
                auto fetch = [&](int i) {
                    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                                 : "=r"(words[4 * i]), "=r"(words[4 * i + 1]), "=r"(words[4 * i + 2]), "=r"(words[4 * i + 3])
                                 : "r"(src + 16u * i) : "memory");
                };
                auto decode = [&](auto block_tag) {                     // K block b of the chunk
                    constexpr int b = decltype(block_tag)::value;
                    const uint32_t *w = words + 7 * b;
                    const uint32_t pool = (w[0] << 16 >> 8) | (((w[0] & 0xff00u) ^ 0x8000u) << 16);
                    // table entry of code byte j
                    auto lookup = [&](int j, uint32_t &e0, uint32_t &e1) {
                        const uint32_t word = w[(2 + j) >> 2];
                        const int k = (2 + j) & 3;
                        uint32_t addr;
                        if (V::WIDE) addr = prmt(word, lane_entry | (j & 1 ? 128u : 0u), 0x7604u | (uint32_t)(k << 4));
                        else addr = prmt(word, 0u, 0x4440u | (uint32_t)k) * 128u + lane_entry;
                        asm("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(e0), "=r"(e1) : "r"(addr));
                    };
                    auto pick = [&](uint32_t sel) { return prmt(pool, 0u, sel); };
                    auto even = [&](uint32_t e0, uint32_t e1, uint32_t &a, uint32_t &c) { a = pick(e0); c = pick(e1); };
                    auto odd = [&](uint32_t e0, uint32_t e1, uint32_t &a, uint32_t &c) {
                        a = pick(V::WIDE ? e0 : prmt(e0, e1, 0x0041));
                        c = pick(V::WIDE ? e1 : prmt(e0, e1, 0x0025));
                    };
                    // trit 4 of an even byte beside trit 0 of the odd byte after it
                    auto straddle = [&](uint32_t p0, uint32_t q0) { return pick(prmt(p0, q0, V::WIDE ? 0x0062 : 0x0042)); };
                    const uint32_t number = (uint32_t)(wave0 + b * width + group);
                    const uint32_t stage = number % RING;
                    const uint32_t a_addr = tmem_lane + (uint32_t)V::kABase + stage * kStageCols;
                    uint32_t m0w, m1w;                                  // byte 12 belongs to both halves
                    {
                        uint32_t v[32];
#pragma unroll
                        for (int a = 0; a < 6; ++a) {
                            uint32_t e0, e1, f0, f1;
                            lookup(2 * a, e0, e1);
                            lookup(2 * a + 1, f0, f1);
                            even(e0, e1, v[5 * a], v[5 * a + 1]);
                            v[5 * a + 2] = straddle(e0, f0);
                            odd(f0, f1, v[5 * a + 3], v[5 * a + 4]);
                        }
                        lookup(12, m0w, m1w);
                        even(m0w, m1w, v[30], v[31]);
                        if (V::kDecodeAhead) wait_read((int)number - RING);
                        else mbar_wait(bar(EMPTY + (int)stage), (number / RING & 1u) ^ 1u, prm.status, dead);
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        tmem_store32(a_addr, v);
                    }
                    {
                        uint32_t v[32], f0, f1;
                        lookup(13, f0, f1);
                        v[0] = straddle(m0w, f0);
                        odd(f0, f1, v[1], v[2]);
#pragma unroll
                        for (int a = 7; a < 12; ++a) {
                            uint32_t e0, e1, g0, g1;
                            lookup(2 * a, e0, e1);
                            lookup(2 * a + 1, g0, g1);
                            even(e0, e1, v[5 * a - 32], v[5 * a - 31]);
                            v[5 * a - 30] = straddle(e0, g0);
                            odd(g0, g1, v[5 * a - 29], v[5 * a - 28]);
                        }
                        uint32_t e0, e1, t0, t1, none;
                        lookup(24, e0, e1);
                        lookup(25, t0, t1);                             // the tail byte's three trits
                        even(e0, e1, v[28], v[29]);
                        v[30] = straddle(e0, t0);
                        odd(t0, t1, v[31], none);
                        tmem_store32(a_addr + 32u, v);
                        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        __syncwarp();
                        const uint32_t full = bar(FULL_A + (int)stage);
                        if (lane == 0) mbar_arrive_leader<CG>(CG == 2 ? leader_addr(full) : full);
                    }
                };
                auto first_block = [&]() {
                    mbar_wait(bar(PACK + warp * V::PACK_STAGES + (int)s), (consumed / V::PACK_STAGES) & 1u, prm.status, dead);
#pragma unroll
                    for (int i = 0; i < (V::kDecodeAhead ? 2 : 4); ++i) fetch(i);
                    decode(std::integral_constant<int, 0>{});
                };
                if (V::kDecodeAhead) {
                    // Not where the group had no chunk for so long that the wait for its ring stage could take a phase for an
                    // older one: then the results, and with them the end of all earlier products, come first.
                    const bool early = done_len == 0 || wave0 + group - RING - seen <= READ_BARS;
#pragma unroll 1
                    for (int turn = 0; turn < 2; ++turn) {
                        if (active && early == (turn == 0)) first_block();
                        if (done_len) {
                            finish(done_tile, done_len, done_part);
                            done_len = 0;
                        }
                    }
                } else if (active) {
                    first_block();
                }
                if (active) {
                    if (V::kDecodeAhead) {
#pragma unroll
                        for (int i = 1; i < 4; ++i) fetch(i);
                    }
                    decode(std::integral_constant<int, 1>{});
#pragma unroll
                    for (int i = 4; i < 7; ++i) fetch(i);
                    ++consumed;
                    __syncwarp();
                    request();
                    decode(std::integral_constant<int, 2>{});
                    decode(std::integral_constant<int, 3>{});
                }
            }
            if (!more) break;
            if (V::kDecodeAhead) { done_tile = tile; done_len = len; done_part = part; }
            else finish(tile, len, part);
        }
    }

    // ---- leave: nothing of this CTA (or of its pair) is in flight any more ---------------------------------------
    __syncwarp();
    if (dead)                                           // a wait ran out: give the copies still in flight time to land
        for (int i = 0; i < 64; ++i) __nanosleep(20000);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (CG == 2) {
        asm volatile("barrier.cluster.arrive.release;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    } else if (CLUSTERED) {
        // Every CTA adds its share of the tile's columns, the parts in the order of their columns of the matrix.
        const int splits = prm.work.splits, tile = prm.work.by_splits.div(slot), part = slot - tile * splits;
        // the tile's counter has no use here; that it is not zero is reported as by the calls that count (a warp with time to spare)
        if (tid == kMmaWarp * 32 && part == 0 && __ldcg(prm.counters + tile) != 0u) atomicExch(prm.status, 8u);
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        const int m0 = token_tile0(tile), all = min(tile_tokens(m0), prm.M - m0), tile_n0 = weight_tile(tile) * kTileW;
        const int first = all * part / splits, quads = (all * (part + 1) / splits - first) * (kTileW / 4);      // four rows of a column each
#pragma unroll 1
        for (int i = tid; i < quads; i += V::kThreads) {
            const int col = first + (i >> 5), m = m0 + col, nq = tile_n0 + (i & 31) * 4;
            if (nq >= prm.N) continue;                  // nothing is read that is not used below
            const uint32_t own = wbase + V::kBAddr + (uint32_t)(col * kTileW + (i & 31) * 4) * 4u;
            float r[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 4
            for (int c = 0; c < splits; ++c) {
                float4 p;
                asm volatile("{\n\t.reg .u32 a;\n\tmapa.shared::cluster.u32 a, %4, %5;\n\t"
                             "ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [a];\n\t}"
                             : "=f"(p.x), "=f"(p.y), "=f"(p.z), "=f"(p.w) : "r"(own), "r"(c) : "memory");
                r[0] += p.x; r[1] += p.y; r[2] += p.z; r[3] += p.w;
            }
            store_quad(r, m, nq);
        }
        // the others' parts have been read (what was read has been used); the results' own way needs no waiting for
        __syncwarp();
        asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    } else {
        __syncthreads();
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (CG == 2)
            asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)V::kTmemCols) : "memory");
        else
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)V::kTmemCols) : "memory");
    }
}

// The token tile names the variant: 16 and 32 run as S, 64 and 128 as L, 256 as P.
int tile_cg(int tile) { return tile > 128 ? 2 : 1; }

struct Tiling {
    int tile, tiles_m, nt;
    WorkSplit work;
    int ctas() const { return work.slots * tile_cg(tile); }
};

// Clusters of `size` CTAs of the clustered kernel for this token tile that run at once.
KernelRecord g_clustered[2];                                    // of variants S and L
int cluster_room(int tile, int size) {
    return tile <= 32 ? clusters_at_once(g_clustered[0], reinterpret_cast<const void *>(tq1_gemm_kernel<VariantS, false, true>),
                                         VariantS::kThreads, VariantS::kSmemBytes, size)
                      : clusters_at_once(g_clustered[1], reinterpret_cast<const void *>(tq1_gemm_kernel<VariantL, false, true>),
                                         VariantL::kThreads, VariantL::kSmemBytes, size);
}

// How the chunks of a shape are dealt out for a given token tile.
Tiling make_tiling(int tile, int M, int N, int K) {
    Tiling t;
    const int cg = tile_cg(tile);
    t.tile = tile;
    t.tiles_m = (M + tile - 1) / tile;
    // equal token tiles: a prompt of 777 tokens is three tiles of 224 and one of 105 rather than three of 256 and one of 9
    const int even = (M + t.tiles_m - 1) / t.tiles_m;
    t.nt = (even + 16 * cg - 1) / (16 * cg) * (16 * cg);
    t.tiles_m = (M + t.nt - 1) / t.nt;
    const long long tiles = (long long)((N + kTileW * cg - 1) / (kTileW * cg)) * t.tiles_m;
    const long long slots = (long long)sm_count() * (tile <= 32 ? 2 : 1) / cg;
    WorkSplit &w = t.work;
    w.chunks = (K / kGroup + kChunkGroups - 1) / kChunkGroups;
    w.total_iters = (int)(tiles * w.chunks);
    w.whole_rounds = w.whole_tiles = 0;
    w.tiles_total = (int)tiles;
    // With more than half as many tiles as slots, cutting every tile in two would need a second wave and one
    // part per tile leaves up to half of the SMs idle: those shapes are shared stream-K fashion as well.
    if (tiles >= slots || (tile > 16 && 2 * tiles > slots)) {
        w.splits = 0;
        w.slots = (int)slots;
        // whole tiles first; what is left over is shared. A share of fewer than two chunks per slot
        // would cost more in partial stores than it balances, so then one round of whole tiles is shared too.
        long long rounds = tiles / slots;
        long long shared = tiles - rounds * slots;
        if (rounds > 0 && shared > 0 && shared * w.chunks < 2 * slots) {
            --rounds;
            shared += slots;
        }
        w.whole_rounds = (int)rounds;
        w.whole_tiles = (int)(rounds * slots);
        w.total_iters = (int)(shared * w.chunks);
        if (shared == 0) w.slots = (int)(tiles < rounds * slots ? (tiles + rounds - 1) / rounds : slots);
        // a slot without a share must not lie between two that share a tile: their sum counts the slots from first to last
        if (rounds == 0 && w.total_iters < w.slots) w.slots = w.total_iters;
    } else {
        int splits = (int)(slots / tiles);
        const int max_splits = w.chunks / 2 > 0 ? w.chunks / 2 : 1;
        if (splits > max_splits) splits = max_splits;
        if (splits > 32) splits = 32;
        w.splits = splits;
        w.slots = (int)tiles * splits;
    }
    w.by_splits.set(w.splits > 0 ? w.splits : 1);
    w.by_chunks.set(w.chunks);
    w.quot = w.total_iters / w.slots;
    w.rem = w.total_iters % w.slots;
    // CTA pairs have one accumulator for most token tiles, and ranges of a whole tile's length side by side would leave a row
    // of tiles in one piece, each under one accumulator (192 tokens of 17408x5120: 4.5e-6 from the FP64 product, spread
    // 4.1e-6). Other ranges come first together, which keeps more of the rest on tile boundaries (1024 tokens of 7168x5120:
    // 67 us, spread 74).
    w.spread = cg == 2 && w.quot + 1 >= w.chunks;
    w.by_slots.set(w.slots);
    return t;
}

// A tile's parts add up in a cluster.
bool clustered(int tile, const WorkSplit &w, const int *rooms = nullptr) {
    return tile <= 128 && w.splits > 1 && w.splits <= kMaxCluster && w.tiles_total <= (rooms ? rooms[w.splits] : cluster_room(tile, w.splits));
}

// Activation rows per tile. Up to 16 rows always take the 16-row tile. Beyond that the choice is one of error as much as of time: it
// says how many columns an accumulator covers. It was made for time, when the parts of a tile met in the workspace: the smallest modelled
// time of launch and pipeline fill, chunks a slot works through (decode, plus products per token), segments it stores, and the sums of
// shared tiles, with constants (us) fitted to the sweep of that form in ternel_b200/dispatch_sweep_b200.json, which tests replay (within
// 10% of the best recorded tile for every case). The times have changed since and the choice has not: the tiles that would be the
// fastest now, by up to 1.7 times, have longer accumulators. g_forced_tile overrides the rule while a sweep is being recorded.
int g_forced_tile = 0;
struct TileCost { int tile; float fixed, chunk, chunk_token, segment, shared_token; };
const TileCost g_tile_costs[5] = {{16, 2.932f, 0.0f, 0.1263f, 1.968f, 0.1093f},
                                  {32, 0.0f, 0.0f, 0.06457f, 1.932f, 0.1664f},
                                  {64, 2.805f, 1.073f, 0.0f, 2.893f, 0.04036f},
                                  {128, 3.198f, 0.8116f, 0.005891f, 2.846f, 0.02803f},
                                  {256, 3.206f, 0.4634f, 0.009061f, 3.616f, 0.03028f}};
float model_us(const TileCost &c, const Tiling &t) {
    const WorkSplit &w = t.work;
    const float shared = (float)w.total_iters / w.slots;        // chunks of shared tiles per slot
    const float chunks = w.splits ? (float)((w.chunks + w.splits - 1) / w.splits)
                                  : (float)w.whole_rounds * w.chunks + ceilf(shared);
    const float segments = w.splits ? 1.0f : (float)w.whole_rounds + (w.total_iters ? shared / w.chunks + 1.0f : 0.0f);
    const bool sums = w.splits ? w.splits > 1 : w.total_iters > 0;
    return c.fixed + chunks * (c.chunk + c.chunk_token * t.nt) + segments * c.segment + (sums ? c.shared_token * t.nt : 0.0f);
}
int token_tile(int M, int N, int K) {
    if (g_forced_tile) return g_forced_tile;
    if (M <= 16) return 16;
    int best = 128;
    float best_cost = 0.0f;
    for (int i = 0; i < 5; ++i) {
        const TileCost &c = g_tile_costs[i];
        if (c.tile > 16 && c.tile >= 4 * M) continue;           // a tile mostly of padding
        const Tiling t = make_tiling(c.tile, M, N, K);
        // whole tiles on less than half of the chip: a narrower tile splits K over the rest, with shorter accumulators
        if (c.tile == 256 && t.work.splits == 1 && 2 * t.ctas() <= sm_count()) continue;
        const float cost = model_us(c, t);
        if (i == 0 || cost < best_cost) { best = c.tile; best_cost = cost; }
    }
    return best;
}
Tiling pick_tiling(int M, int N, int K) { return make_tiling(token_tile(M, N, K), M, N, K); }

size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

template <class V, bool GATED, bool CLUSTERED>
int launch_kernel(KernelRecord &record, const CUtensorMap &wmap, const CUtensorMap &xmap, const GemmParams &prm, int ctas, cudaStream_t stream) {
    auto kern = tq1_gemm_kernel<V, GATED, CLUSTERED>;
    const cudaError_t e = opt_in(record, reinterpret_cast<const void *>(kern), V::kSmemBytes, CLUSTERED);
    if (e != cudaSuccess) return cuda_fail(e, "tq1_linear_f16: shared memory opt-in (GEMM)");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(V::kThreads);
    cfg.dynamicSmemBytes = V::kSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = CLUSTERED ? (unsigned)prm.work.splits : V::CG;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = V::CG > 1 || CLUSTERED ? 2 : 1;
    const cudaError_t err = cudaLaunchKernelEx(&cfg, kern, wmap, xmap, prm);
    if (err == cudaSuccess && stream_captured(stream)) note_captured_kernel(stream);
    return err == cudaSuccess ? TQ1_OK : cuda_fail(err, "tq1_linear_f16: GEMM launch");
}

template <class V, bool GATED>
int launch_variant(const CUtensorMap &wmap, const CUtensorMap &xmap, GemmParams &prm, int ctas, cudaStream_t stream) {
    const int stages = (int)(V::kBRoom / ((uint32_t)prm.b_rows * 256u));
    prm.b_stages = stages < V::RING ? stages : V::RING;
    static KernelRecord record, in_clusters;
    if constexpr (V::CG == 1) {
        static_assert(V::MAX_COLS * kTileW * 4 <= V::kBRoom, "a part lies where the activations were");
        // in clusters, where all of them run at once
        if (clustered(V::G == 2 ? 32 : 128, prm.work))
            return launch_kernel<V, GATED, true>(in_clusters, wmap, xmap, prm, ctas, stream);
    }
    return launch_kernel<V, GATED, false>(record, wmap, xmap, prm, ctas, stream);
}

}  // namespace

int gemm_tc_force_tile(int nt) {
    if (nt != 0 && nt != 16 && nt != 32 && nt != 64 && nt != 128 && nt != 256) return TQ1_ERR_INVALID;
    g_forced_tile = nt;
    return TQ1_OK;
}

bool gemm_tc_forced() { return g_forced_tile != 0; }

// What draws the line between this kernel and the slice kernel, whose sums have a third to a tenth of the error: times fitted to 1022
// calls behind another kernel when parts still met in the workspace. The line is kept for the error: since a cluster adds the parts this
// kernel would be the faster one for 39 of 380 calls of nine to sixteen tokens that are left to the other, by 11% on average.
float gemm_tc_few_us(int N, int K) {
    const Tiling t = make_tiling(16, 16, N, K);
    const WorkSplit &w = t.work;
    const int tiles = w.splits ? 1 : w.whole_rounds;
    const int chunks = w.splits ? (w.chunks + w.splits - 1) / w.splits : tiles * w.chunks + (w.total_iters + w.slots - 1) / w.slots;
    return 5.32f + 1.084f * (float)chunks + (t.ctas() > sm_count() ? 1.22f * (float)tiles : 0.0f) +
           (w.splits > 1 ? 0.69f + 0.263f * (float)w.splits : 0.0f) + (!w.splits && w.total_iters ? 0.74f : 0.0f) +
           66.9e-9f * (float)N * (float)K;
}

void gemm_tc_plan(int M, int N, int K, int *tile, int *ctas, int *parts) {
    const Tiling t = pick_tiling(M, N, K);
    *tile = t.tile;
    *ctas = t.ctas();
    *parts = t.work.splits;
}

bool gemm_tc_layout(int M, int N, int K, const int *rooms, CallLayout *layout) {
    if (!gemm_tc_shape_ok(M, N, K)) return false;
    const Tiling t = pick_tiling(M, N, K);
    *layout = {clustered(t.tile, t.work, rooms) ? t.work.splits : 1, t.work.splits, 0, t.work.tiles_total, true};
    return true;
}

bool gemm_tc_shape_ok(int M, int N, int K) { return M >= 2 && N >= 1 && K % (kChunkGroups * kGroup) == 0; }

size_t gemm_tc_workspace_bytes(int M, int N, int K) {
    const Tiling t = pick_tiling(M, N, K);
    return kWsScratchOffset + align256((size_t)2 * t.ctas() * t.nt * kTileW * sizeof(float));
}

// The largest such size over all tiles, N and K, and over all smaller batches: token columns in flight on one SM are at most
// 32 (two 16-token tiles), two 32-token tiles or one tile of the batch's length.
size_t gemm_tc_workspace_bound(int M) {
    const int columns = M <= 16 ? 32 : M <= 64 ? 64 : M >= 256 ? 256 : (M + 31) / 32 * 32;
    return kWsScratchOffset + align256((size_t)2 * sm_count() * columns * kTileW * sizeof(float));
}

int launch_gemm_tc(const uint8_t *blocks, const __half *x, void *y, bool y_f32, int M, int N, int K,
                   void *workspace, cudaStream_t stream, bool swiglu) {
    EncodeTiledFn encode = encode_tiled_fn();
    if (!encode) return fail(TQ1_ERR_CUDA, "tq1_linear_f16: cuTensorMapEncodeTiled is unavailable");
    unsigned char *ws = static_cast<unsigned char *>(workspace);
    const Tiling t = pick_tiling(M, N, K);
    const int cg = tile_cg(t.tile);
    GemmParams prm;
    prm.y = y;
    prm.partials = reinterpret_cast<float *>(ws + kWsScratchOffset);
    prm.counters = reinterpret_cast<unsigned *>(ws + kWsCounterOffset);
    prm.status = reinterpret_cast<unsigned *>(ws);
    prm.M = M;
    prm.N = N;
    prm.groups = K / kGroup;
    prm.tiles_m = t.tiles_m;
    prm.by_tiles_m.set(t.tiles_m);
    prm.nt = t.nt;
    prm.b_rows = t.nt / cg;
    const int acc_area = t.tile <= 32 ? VariantS::ACC_COLS : t.tile <= 128 ? VariantL::ACC_COLS : VariantP::ACC_COLS;
    prm.accs = 4 * t.nt <= acc_area ? 4 : 2 * t.nt <= acc_area ? 2 : 1;       // a segment has at least four K blocks
    prm.acc_cols = acc_area / prm.accs;
    prm.work = t.work;
    prm.y_f32 = y_f32 ? 1 : 0;
    const uintptr_t y_addr = reinterpret_cast<uintptr_t>(y);
    prm.pair_y = N % 2 == 0 && (y_addr & 3) == 0 ? 1 : 0;
    prm.quad_y = N % 4 == 0 && (y_addr & ((y_f32 ? 16 : 8) / (swiglu ? 2 : 1) - 1)) == 0 ? 1 : 0;

    CUtensorMap wmap, xmap;
    const cuuint32_t estr[2] = {1, 1};
    {
        const cuuint64_t row_bytes = (cuuint64_t)(K / kGroup) * kBlockBytes;
        const cuuint64_t dims[2] = {row_bytes, (cuuint64_t)N};
        const cuuint64_t strides[1] = {row_bytes};
        const cuuint32_t box[2] = {kChunkBytes, 32};
        CUresult res = encode(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t *>(blocks), dims, strides,
                              box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                              // L2 is asked for 112-byte pieces of rows; for few tokens, where the weights are most of the traffic,
                              // 64-byte fetches bring in less that is not used (8 tokens, 34816x5120: 27.4 -> 26.8 us,
                              // 5120x17408: 19.9 -> 19.3). From 33 tokens on 256 bytes are 0.7% faster.
                              t.tile <= 32 ? CU_TENSOR_MAP_L2_PROMOTION_L2_64B : CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (res != CUDA_SUCCESS) return fail(TQ1_ERR_CUDA, "tq1_linear_f16: weight tensor map failed (%d)", (int)res);
    }
    {
        const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)M};
        const cuuint64_t strides[1] = {(cuuint64_t)K * sizeof(__half)};
        const cuuint32_t box[2] = {64, (cuuint32_t)prm.b_rows};
        CUresult res = encode(&xmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half *>(x), dims, strides, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (res != CUDA_SUCCESS)
            return fail(TQ1_ERR_CUDA, "tq1_linear_f16: activation tensor map failed (%d)", (int)res);
    }
    const auto launch = [&](auto gated) {
        constexpr bool GATED = decltype(gated)::value;
        return t.tile <= 32    ? launch_variant<VariantS, GATED>(wmap, xmap, prm, t.ctas(), stream)
               : t.tile <= 128 ? launch_variant<VariantL, GATED>(wmap, xmap, prm, t.ctas(), stream)
                               : launch_variant<VariantP, GATED>(wmap, xmap, prm, t.ctas(), stream);
    };
    return swiglu ? launch(std::true_type{}) : launch(std::false_type{});
}

}  // namespace tq1
