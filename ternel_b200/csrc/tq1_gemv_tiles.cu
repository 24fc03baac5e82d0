// One or two activation rows for widths that are multiples of 512, as a call of its own: the exact arithmetic of the chain kernel
// (tq1_gemv_chain.cu) with a row's whole sum inside a CTA, or a cluster.
//
// The chain kernel numbers its units chunk after chunk, so that any number of them falls evenly on 148 CTAs; a row's chunks then
// meet through workspace slots, and a matrix of canonical blocks is read in row pieces of 112 bytes. For a list of links that
// is what keeps the GPU busy; for one product it costs two round trips through L2, a 64 KB table from memory, and a third more
// DRAM traffic than there are weights. Here
//
//   warp      keeps the digit planes of one 512-column chunk (of one activation row) in registers and streams 16-row tiles past
//             it: one unit of the chain kernel per tile
//   set       as many warps as the CTA's K range has chunks (times activation rows); sets take turns on the row tiles. A tile
//             arrives by one TMA box, 16 rows of the whole K range: rows of a matrix are neighbours, so a CTA reads DRAM in
//             pieces of 18 KB (5120 columns). Rows lie an odd number of 16-byte units apart: no bank conflicts.
//   sums      the chunks' partial sums of a tile meet in shared memory; two tiles later one of the set's warps, in turn, adds them
//             in the chain kernel's order (even chunks, odd chunks, both), so results are the same to the bit
//   cluster   2, 4 or 8 CTAs split K where one CTA has no warps for it; partial sums go to the CTA that adds a tile's through
//             distributed shared memory
//
// Where even four CTAs would not do, or do no better, the chain kernel takes the call (not_behind_chain).
//
// The table (256 entries, 32 copies each) is worked out by the CTA's warps, four entries per instruction.
//
// What bounds it: many rows, the loop of the units, 105 clocks of an SM each (76 wavefronts of shared memory, about 330 instructions
// on four issue ports, twenty warps to hide the latencies); few rows, the chain set-up - activations - planes - first tile - sums
// (7000 clocks behind another kernel, a third of it the planes). The chain kernel for one link and this one, FP32 results, weights
// out of HBM, calls in a row (us): 1024x5120 5.8, 3.4; 4096x4096 6.3, 4.2; 5120x5120 7.3, 5.6; 17408x5120 11.4, 9.4; 151936x5120 52.6,
// 43.6; 5120x17408 11.5, 11.3; 48x512 4.4, 2.1. Two activation rows: 1024x5120 9.0, 4.8; 17408x5120 19.1, 14.7; 5120x17408 19.4, 16.5.
// Taken back on the way: the next tile asked for when sums are added up, after the tile's own products (no distance left: 151936x5120
// 71.5 us, before them 50.3); loop bookkeeping left to kernel parameters and divisions (50.3, 45.8); a thread's barriers and a
// cluster barrier around the sums of split K (5120x17408 12.2, 11.3 with st.async and a barrier per tile).
#include <cuda.h>
#include <math.h>

#include <type_traits>

#include "tq1_decode.cuh"
#include "tq1_gemv_unit.cuh"

namespace tq1 {

namespace {

constexpr int kMaxWarps = 20;                                   // 96 registers each
constexpr uint32_t kWindow = 1024;                              // shared-window address of dynamic shared memory
constexpr uint32_t kTableAddr = kWindow;                        // 256 entries of 256 bytes, of which 128 hold an entry's copies
constexpr uint32_t kTableBytes = 65536;
constexpr uint32_t kBarAddr = kTableAddr + kTableBytes;
constexpr uint32_t kConstAddr = kBarAddr + 2048;                // constants of the groups
constexpr uint32_t kDataAddr = kConstAddr + kMaxWarps * kChunkGroups * sizeof(GroupConst);      // sums, ring
constexpr uint32_t kWindowEnd = 227 * 1024;
constexpr int kMinWarps = 8;                                    // fewer would be long at the table
constexpr int kLag = 2;                                         // a tile is added up while the second one after it is decoded
constexpr int kBufs = 2 * kLag;
constexpr int kMaxOwn = 128;                                    // tiles that a CTA of a cluster adds up
constexpr int kMaxTokens = 2;
// The barriers: sums; ring; where clusters split K, one for each tile that a CTA adds up.
constexpr int kRingBars = kMaxWarps * kBufs, kTileBars = 256 - kMaxOwn;
constexpr int kMaxStages = (kLag + 1) * kMaxWarps, kMaxStagesSplit = 48;
static_assert(kRingBars + kMaxStages <= 256 && kRingBars + kMaxStagesSplit <= kTileBars, "barrier area of 2048 bytes");

struct TileParams {
    const __half *x;                                            // [tokens][chunks * 512]
    void *y;
    unsigned *status;
    int N, chunks;
    int tiles, clusters;                                        // row tiles, clusters of the grid
    int split_log, slices, subsets;                             // CTAs of a cluster; chunks of a CTA at most; sets of warps
    int stages, early, pitch;                                   // ring stages; those that are filled before the planes; bytes from row to row
    uint32_t plane_addr, xchg_addr, sums_addr, ring_addr;       // the scratch (planes, exchange) lies where the last stages are
    int y_f32, swiglu;
};

// The partial sums of one chunk for rows g and g + 8 of a tile, in the lanes with q = 0.
template <bool BAD>
__device__ __forceinline__ void chunk_sums(uint32_t a1, uint32_t row8, uint32_t lane_base, const uint32_t (&breg)[2 * kRegsPerSub],
                                           const int (&gsum)[2], const float (&gpow)[2], const int (&gbad)[2], float &acc1,
                                           float &acc2) {
    asm volatile("" : "+r"(a1));                              // no load before the wait for the tile
    const uint32_t a2 = a1 + row8;
    acc1 = acc2 = 0.0f;
#pragma unroll
    for (int sub = 0; sub < 2; ++sub) {
        const uint32_t w1a = sub ? lds_off<28>(a1) : lds_off<0>(a1), w1b = sub ? lds_off<32>(a1) : lds_off<4>(a1);
        const uint32_t w1c = sub ? lds_off<36>(a1) : lds_off<8>(a1), w1d = sub ? lds_off<40>(a1) : lds_off<12>(a1);
        const uint32_t w2a = sub ? lds_off<28>(a2) : lds_off<0>(a2), w2b = sub ? lds_off<32>(a2) : lds_off<4>(a2);
        const uint32_t w2c = sub ? lds_off<36>(a2) : lds_off<8>(a2), w2d = sub ? lds_off<40>(a2) : lds_off<12>(a2);
        uint32_t r1[kRegsPerSub], r2[kRegsPerSub];
        decode_stream<kTableAddr>(w1a, w1b, w1c, w1d, lane_base, r1);
        decode_stream<kTableAddr>(w2a, w2b, w2c, w2d, lane_base, r2);
        int acc[4];
        mma_bytes<true, true>(acc, r1[0], r2[0], r1[1], r2[1], breg[sub * kRegsPerSub + 0], breg[sub * kRegsPerSub + 1]);
#pragma unroll
        for (int r = 2; r < 14; r += 2) mma_bytes<true, false>(acc, r1[r], r2[r], r1[r + 1], r2[r + 1], breg[sub * kRegsPerSub + r], breg[sub * kRegsPerSub + r + 1]);
        mma_bytes<false, false>(acc, r1[14], r2[14], r1[15], r2[15], breg[sub * kRegsPerSub + 14], breg[sub * kRegsPerSub + 15]);
        mma_bytes<false, false>(acc, r1[16], r2[16], r1[17], r2[17], breg[sub * kRegsPerSub + 16], breg[sub * kRegsPerSub + 17]);
        const uint32_t pair1 = (uint32_t)acc[0] + ((uint32_t)acc[1] << 8);
        const uint32_t pair2 = (uint32_t)acc[2] + ((uint32_t)acc[3] << 8);
        const uint32_t hi1 = __shfl_down_sync(0xffffffffu, pair1, 1);
        const uint32_t hi2 = __shfl_down_sync(0xffffffffu, pair2, 1);
        const int s1 = (int)((pair1 + (hi1 << 16) - (uint32_t)gsum[sub]) * 0x781948b1u);
        const int s2 = (int)((pair2 + (hi2 << 16) - (uint32_t)gsum[sub]) * 0x781948b1u);
        float dot1 = (float)s1 * gpow[sub], dot2 = (float)s2 * gpow[sub];
        if (BAD && gbad[sub]) {                                 // +-n of a group's n infinite products, or NaN
            const float inf = __int_as_float(0x7f800000), nan = __int_as_float(0x7fffffff);
            dot1 = s1 == gbad[sub] ? inf : s1 == -gbad[sub] ? -inf : nan;
            dot2 = s2 == gbad[sub] ? inf : s2 == -gbad[sub] ? -inf : nan;
        }
        acc1 = fmaf(__half2float(__ushort_as_half((unsigned short)(w1a & 0xffffu))), dot1, acc1);
        acc2 = fmaf(__half2float(__ushort_as_half((unsigned short)(w2a & 0xffffu))), dot2, acc2);
    }
    acc1 += __shfl_down_sync(0xffffffffu, acc1, 2);
    acc2 += __shfl_down_sync(0xffffffffu, acc2, 2);
}

// Adds a tile's partial sums (16 floats per chunk from `parts` on) and stores the results of its rows.
template <int TOKENS>
__device__ __forceinline__ void finish_tile(const TileParams &prm, const float *parts, int tile, int token, int lane) {
    const int r = lane & 15, hf = lane >> 4;
    float total = 0.0f;
#pragma unroll 4
    for (int c = hf; c < prm.chunks; c += 2) total += parts[c * kTileRows + r];
    total += __shfl_xor_sync(0xffffffffu, total, 16);
    int row = tile * kTileRows + r, n = prm.N;
    bool writer = hf == 0 && row < n;
    if (prm.swiglu) {                                           // (gate, up) row pairs
        total = swiglu_f32(total, __shfl_down_sync(0xffffffffu, total, 1));
        writer = writer && (r & 1) == 0 && row + 1 < n;
        row >>= 1;
        n >>= 1;
    }
    const size_t o = (size_t)token * n + row;
    if (writer && TQ1_IN_BOUNDS(o, (size_t)TOKENS * n, 90u)) {
        if (prm.y_f32) static_cast<float *>(prm.y)[o] = total;
        else static_cast<__half *>(prm.y)[o] = __float2half_rn(total);
    }
}

// SPLIT: clusters split K.
template <bool SPLIT, int TOKENS>
__global__ void __launch_bounds__(32 * kMaxWarps, 1)
tiles_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ TileParams prm) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const uint32_t window = (uint32_t)__cvta_generic_to_shared(smem);
    const uint32_t base = window - kWindow;                     // zero, or what names this CTA of a cluster
    if ((base & 0x00ffffffu) != 0u) {                           // the fixed window addresses do not hold
        if (threadIdx.x == 0) atomicExch(prm.status, 2u);
        return;
    }
    auto at = [&](uint32_t addr) { return smem + (addr - kWindow); };
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int warps = blockDim.x >> 5;
    const int split_log = SPLIT ? prm.split_log : 0, split = 1 << split_log, rank = blockIdx.x & (split - 1), cluster = blockIdx.x >> split_log;
    const int chunk_lo = prm.chunks * rank >> split_log, n_slices = (prm.chunks * (rank + 1) >> split_log) - chunk_lo;
    const int tile_lo = (int)((long long)cluster * prm.tiles / prm.clusters);
    const int n_tiles = (int)((long long)(cluster + 1) * prm.tiles / prm.clusters) - tile_lo;
    const int set_warps = n_slices * TOKENS;                // of this CTA's sets
    const uint32_t stage_bytes = (uint32_t)(kTileRows * prm.pitch);
    auto sum_bar = [&](int s) { return base + kBarAddr + 8u * (uint32_t)s; };
    auto full_bar = [&](int s) { return base + kBarAddr + 8u * (uint32_t)(kRingBars + s); };
    auto tile_bar = [&](int s) { return base + kBarAddr + 8u * (uint32_t)(kTileBars + s); };
    const int own_tiles = (n_tiles - rank + split - 1) >> split_log;

    // ---- set-up that depends on no earlier kernel ---------------------------------------------------------------
    int *xchg = reinterpret_cast<int *>(at(prm.xchg_addr)) + warp * 2 * kGroup;
    if (tid < prm.stages) mbar_init(full_bar(tid), 1);
    if (tid < kBufs * prm.subsets) mbar_init(sum_bar(tid), (uint32_t)set_warps);
    if (SPLIT && tid < own_tiles) mbar_init(tile_bar(tid), 1);
    if (tid < max(max(prm.stages, kBufs * prm.subsets), SPLIT ? own_tiles : 0)) {
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (SPLIT && tid < own_tiles) mbar_expect_tx(tile_bar(tid), (uint32_t)(TOKENS * prm.chunks * kTileRows * 4));
    if (tid == 32) asm volatile("prefetch.tensormap [%0];" ::"l"(&wmap) : "memory");
    const int word_x = chunk_lo * (kChunkBytes / 8);            // the map's elements are 8 bytes
    if (warp == warps - 1 && elect_one())                       // the first tiles: into L2 (a hint, whatever they hold by now)
        for (int i = 0; i < min(prm.early, n_tiles); ++i)
            asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];"
                         ::"l"(&wmap), "r"(word_x), "r"((tile_lo + i) * kTileRows) : "memory");
    // what no activation is paired with (scales, half of the word that two lanes share) stays zero
    for (int i = tid; i < set_warps * (kPlaneChunk / 16); i += blockDim.x)
        reinterpret_cast<uint4 *>(at(prm.plane_addr))[i] = make_uint4(0u, 0u, 0u, 0u);
    // An entry: trits 0..3 of the byte as signed bytes; 13 bytes past 242 decode to zeros. v / 3 = 171 v >> 9 for v < 256.
    for (int v = 4 * warp + (lane >> 3); v < 256; v += 4 * warps) {
        uint32_t entry = 0, rest = (uint32_t)v;
#pragma unroll
        for (int d = 0; d < 4; ++d) {
            const uint32_t third = rest * 171u >> 9;
            entry |= ((rest - 3u * third - 1u) & 0xffu) << (8 * d);
            rest = third;
        }
        if (v > 242) entry = 0u;
        *reinterpret_cast<uint4 *>(at(kTableAddr) + v * 256 + (lane & 7) * 16) = make_uint4(entry, entry, entry, entry);
    }
    __syncthreads();
    if (SPLIT) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");     // this CTA may be written into
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");

    bool dead = false;
    // set, chunk of the CTA and activation row of this warp
    const int subset = warp / set_warps, in_set = warp - subset * set_warps;
    const int token = TOKENS > 1 && in_set >= n_slices ? 1 : 0, slice = in_set - token * n_slices;
    const bool works = subset < prm.subsets;
    auto fetch = [&](int i, int stage) {                        // called by one thread
        mbar_expect_tx(full_bar(stage), stage_bytes);
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                     ::"r"(base + prm.ring_addr + (uint32_t)stage * stage_bytes), "l"(&wmap), "r"(word_x),
                       "r"((tile_lo + i) * kTileRows), "r"(full_bar(stage)) : "memory");
    };

    // ---- digit planes of the CTA's K range ------------------------------------------------------------------------
    GroupConst *consts = reinterpret_cast<GroupConst *>(at(kConstAddr));
    const int groups = n_slices * kChunkGroups;                 // of one activation row
    // Every warp has all its activations (of at most four groups: there are four warps to sixteen groups) on their way before the
    // weights are asked for: the other way round the few bytes queue behind megabytes.
    uint2 raw[kChunkGroups];
#pragma unroll
    for (int k = 0; k < kChunkGroups; ++k) {
        raw[k] = make_uint2(0u, 0u);
        const int j = warp + k * warps, t = TOKENS > 1 && j >= groups ? 1 : 0;
        if (j < groups * TOKENS)
            raw[k] = *reinterpret_cast<const uint2 *>(prm.x + (size_t)t * prm.chunks * kChunkCols + (size_t)chunk_lo * kChunkCols +
                                                      (size_t)(j - t * groups) * kGroup + 4 * lane);
    }
    if (warp == warps - 1 && elect_one())
        for (int i = 0; i < min(prm.early, n_tiles); ++i) fetch(i, i);
    __syncwarp();
#pragma unroll 1
    for (int j = warp; j < groups * TOKENS; j += 2 * warps) {
        float xv[2][4];
        unsigned char *planes[2];
        GroupConst *results[2];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const __half2 lo = reinterpret_cast<const __half2 &>(raw[n].x), hi = reinterpret_cast<const __half2 &>(raw[n].y);
            xv[n][0] = __low2float(lo); xv[n][1] = __high2float(lo); xv[n][2] = __low2float(hi); xv[n][3] = __high2float(hi);
            const int group = j + n * warps;
            planes[n] = at(prm.plane_addr) + (group >> 2) * kPlaneChunk + plane_group(group & 3);
            results[n] = consts + group;
            raw[n] = raw[n + 2];
        }
        prepare_groups<2, true>(xv, j + warps < groups * TOKENS ? 2 : 1, lane, xchg, planes, results);
        __syncwarp();
    }
    __syncthreads();

    const int g = lane >> 2, q = lane & 3, cls = q >> 1, h = q & 1;
    uint32_t breg[2 * kRegsPerSub];
    int gsum[2], gbad[2];
    float gpow[2];
    load_planes(breg, base + prm.plane_addr + (uint32_t)in_set * kPlaneChunk, lane);
#pragma unroll
    for (int sub = 0; sub < 2; ++sub) {
        const GroupConst gc = consts[in_set * kChunkGroups + sub + 2 * cls];
        gsum[sub] = gc.sum;
        gpow[sub] = gc.pow;
        gbad[sub] = gc.bad;
    }
    if (prm.early < min(prm.stages, n_tiles)) {                 // the other stages: their place may have been the scratch
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (warp == warps - 1 && elect_one())
            for (int i = prm.early; i < min(prm.stages, n_tiles); ++i) fetch(i, i);
        __syncwarp();
    }

    if (SPLIT) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (works) {
        const bool bad = __any_sync(0xffffffffu, (gbad[0] | gbad[1]) != 0);
        const uint32_t lane_base = base | (uint32_t)lane * 4u, row8 = 8u * (uint32_t)prm.pitch;
        const uint32_t lane_src = base + prm.ring_addr + (uint32_t)(g * prm.pitch + slice * kChunkBytes + 2 * cls * kBlockBytes + 12 * h);
        const uint32_t own_bar = sum_bar(kBufs * subset);
        const int buf_floats = TOKENS * prm.chunks * kTileRows;             // a tile's partial sums
        float *sums = reinterpret_cast<float *>(at(prm.sums_addr));
        float *parts = sums + (size_t)subset * kBufs * buf_floats;              // split K: not used, all tiles are kept
        const int part = (token * prm.chunks + chunk_lo + slice) * kTileRows + g;

        auto run = [&](auto bad_tag) {
            constexpr bool BAD = decltype(bad_tag)::value;
            int stage = subset, k = 0, turn = in_set;           // turn: tiles of the set until this warp adds one up
            uint32_t phase = 0;
            auto wait_sums = [&](int j) {                       // of the set's j-th tile
                mbar_wait(own_bar + 8u * (uint32_t)(j % kBufs), (uint32_t)(j / kBufs) & 1u, prm.status, dead);
            };
            auto add_up = [&](int j) {
                wait_sums(j);
                const int i = subset + j * prm.subsets;
                if (i + prm.stages < n_tiles && elect_one() && !dead) {         // the tile's stage is free
                    const int freed = stage - kLag * prm.subsets;
                    fetch(i + prm.stages, freed < 0 ? freed + prm.stages : freed);
                }
                __syncwarp();
                if (!SPLIT) {
#pragma unroll
                    for (int t = 0; t < TOKENS; ++t)
                        finish_tile<TOKENS>(prm, parts + (j % kBufs) * buf_floats + t * prm.chunks * kTileRows, tile_lo + i, t, lane);
                }
            };
            for (int i = subset; i < n_tiles; i += prm.subsets, ++k) {
                if (k >= kLag && turn-- == 0) {
                    turn = set_warps - 1;
                    add_up(k - kLag);
                }
                mbar_wait(full_bar(stage), phase, prm.status, dead);
                float acc1, acc2;
                chunk_sums<BAD>(lane_src + (uint32_t)stage * stage_bytes, row8, lane_base, breg, gsum, gpow, gbad, acc1, acc2);
                stage += prm.subsets;
                if (stage >= prm.stages) { stage -= prm.stages; phase ^= 1u; }
                // That every warp has stored its sums of the tile kLag before this one also says that the sums of the one kLag
                // before that are added up, whose buffer this tile takes.
                if (k >= kLag) wait_sums(k - kLag);
                if (q == 0) {
                    if (!SPLIT) {
                        float *dst = parts + (k % kBufs) * buf_floats + part;
                        dst[0] = acc1;
                        dst[8] = acc2;
                    } else {                                    // to CTA i % split of the cluster
                        uint32_t dst, bar;
                        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst)
                                     : "r"(base + prm.sums_addr + 4u * (uint32_t)((i >> split_log) * buf_floats + part)), "r"(i & (split - 1)));
                        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(bar) : "r"(tile_bar(i >> split_log)), "r"(i & (split - 1)));
                        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%3];\n\t"
                                     "st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0+32], %2, [%3];"
                                     ::"r"(dst), "r"(__float_as_uint(acc1)), "r"(__float_as_uint(acc2)), "r"(bar) : "memory");
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(own_bar + 8u * (uint32_t)(k % kBufs));
            }
            for (int j = k < kLag ? 0 : k - kLag; j < k; ++j)
                if (turn-- == 0) {
                    turn = set_warps - 1;
                    add_up(j);
                }
        };
        if (bad) run(std::true_type{});
        else run(std::false_type{});
    }
    if (dead)                                                   // a wait ran out: give the copies still in flight time to land
        for (int i = 0; i < 64; ++i) __nanosleep(20000);
    if (SPLIT) {                                                // the cluster's sums of this CTA's tiles; when they are there nobody writes here any more
        const float *sums = reinterpret_cast<const float *>(at(prm.sums_addr));
        for (int j = warp; j < own_tiles * TOKENS; j += warps) {
            mbar_wait(tile_bar(j / TOKENS), 0, prm.status, dead);
            finish_tile<TOKENS>(prm, sums + (size_t)j * prm.chunks * kTileRows, tile_lo + rank + (j / TOKENS << split_log), j % TOKENS, lane);
        }
        if (dead) stay_with_cluster();
    }
}

// ---- host ---------------------------------------------------------------------------------------------------------
struct TilePlan {
    bool ok, faster;                                            // fits; and is not behind the chain kernel
    float us;
    int split_log, slices, subsets, clusters, stages, pitch;
    int early;
    uint32_t plane_addr, xchg_addr, sums_addr, ring_addr, end;
};

KernelRecord g_records[2][kMaxTokens];                          // [clusters split K][activation rows - 1]
typedef void (*TileKernel)(CUtensorMap, TileParams);
TileKernel kernel_of(bool split, int tokens) {
    return split ? (tokens > 1 ? tiles_kernel<true, 2> : tiles_kernel<true, 1>) : (tokens > 1 ? tiles_kernel<false, 2> : tiles_kernel<false, 1>);
}

// Modelled time (us) by which a K split is chosen: launch and set-up, a cluster's barriers, what the SM works through, or where
// there are few warps what one of them does one tile after the other. Against every split that fits, in 140 calls of 64 to 34816 rows
// and 1024 to 17408 columns: from 4096 rows on 1.6% above the best on average and 12% at most, with 1024 and 2048 rows 11%, with fewer
// 29%. Small matrices are split too little (64x9216 4.5 us, with eight CTAs to a tile 2.4; 1024x8192 4.4 and 3.2).
float tile_us(int split_log, int set_warps, int subsets, int per_cluster) {
    const float sm = 0.062f * (float)(per_cluster * set_warps), chain = 0.75f * (float)((per_cluster + subsets - 1) / subsets);
    return 3.0f + (split_log ? 1.2f : 0.0f) + (sm > chain ? sm : chain);
}

// Columns that only four or eight CTAs have room for: their clusters leave SMs idle (132 and 120 work), and a CTA has ten to twenty
// warps as the columns come out, while the chain kernel's units fall evenly on 148 times sixteen. One row, the chain kernel and this
// one (us): 20000x20480 30.9, 28.5; 34816x18944 42.1, 43.6; 9000x25600 20.3, 22.1; 20000x25600 35.9, 41.0; 34816x32768 75.4, 100; two
// rows: 5000x25600 25.1, 23.9; 20000x25600 66, 78. Times fitted to 283 such calls (within 6 and 4%, 2-norm): what they choose is 0.4%
// above the better one on average; of 51 calls that this kernel lost 3 to 33% with three are left, of at most 5%, and ten are given up
// that it was 3 to 13% faster with. Narrower matrices are its own: with none of 208 it was behind by more than 2.2%.
bool not_behind_chain(const TilePlan &p, int tokens, int tiles, int chunks) {
    const float per = (float)((tiles + p.clusters - 1) / p.clusters), units = (float)(tiles * (long long)chunks) / (float)sm_count();
    const float turns = ceilf(per / (float)p.subsets), other = (float)(tokens - 1);
    const float own = 4.35f + per * (float)(p.slices * tokens) * (0.054f - 0.005f * other) + 0.22f * turns;
    const float chain = 5.4f + 2.4f * other + (float)tokens * (0.0707f * units + 0.0186f * (float)chunks);
    return own <= chain;
}

TilePlan tile_plan(int tokens, int N, int K, const int *rooms = nullptr) {
    TilePlan best = {};
    const int chunks = K / kChunkCols, tiles = (N + kTileRows - 1) / kTileRows;
    bool narrow = false;                                        // two CTAs have room for the columns
    for (int log = 0; log <= 3; ++log) {
        const int split = 1 << log;
        TilePlan p = {};
        p.split_log = log;
        p.slices = (chunks + split - 1) / split;
        const int set_warps = p.slices * tokens;
        p.pitch = p.slices * kChunkBytes;
        if (p.pitch / 16 % 2 == 0) p.pitch += 16;
        if (chunks < split || set_warps > kMaxWarps || p.pitch / 8 > 256) continue;      // a box has at most 256 elements a row
        const auto subsets_for = [&](int per) { return kMaxWarps / set_warps < per ? kMaxWarps / set_warps : per; };
        // how many clusters run at once is asked of the driver (milliseconds, the first time) only where this split could win
        const int hope = (tiles + sm_count() / split - 1) / (sm_count() / split);
        if (best.ok && tile_us(log, set_warps, subsets_for(hope), hope) >= best.us) continue;
        const int room = rooms ? rooms[split]
                               : clusters_at_once(g_records[log > 0][tokens - 1], reinterpret_cast<const void *>(kernel_of(log > 0, tokens)),
                                                  32 * kMaxWarps, kWindowEnd - kWindow, split);
        if (room < 1) continue;
        p.clusters = tiles < room ? tiles : room;
        const int per = (tiles + p.clusters - 1) / p.clusters;
        p.subsets = subsets_for(per);
        const auto aligned = [](size_t bytes) { return (uint32_t)((bytes + 127) / 128 * 128); };
        p.sums_addr = kDataAddr;
        const size_t kept = log ? (size_t)(per + split - 1) / split : (size_t)p.subsets * kBufs;
        const size_t sum_bytes = kept * tokens * chunks * kTileRows * 4;
        if (sum_bytes > kWindowEnd || (log && (per + split - 1) / split > kMaxOwn)) continue;
        p.ring_addr = p.sums_addr + aligned(sum_bytes);
        const uint32_t stage_bytes = (uint32_t)(kTileRows * p.pitch);
        const uint32_t plane_bytes = aligned((size_t)set_warps * kPlaneChunk), scratch = plane_bytes + kMaxWarps * 2 * kGroup * 4;
        if (p.ring_addr + scratch + stage_bytes > kWindowEnd) continue;
        const auto stages_in = [&](uint32_t end) {
            const int n = (int)((end - p.ring_addr) / stage_bytes), most = log ? kMaxStagesSplit : kMaxStages;
            return n > most ? most : n;
        };
        p.stages = stages_in(kWindowEnd) < per ? stages_in(kWindowEnd) : per;
        if (p.stages < per) {
            // A stage is asked for again kLag turns of its set after it was read. And it belongs to one set: a wait for a barrier's
            // parity tells a phase from the one before it only, so who waits has to have seen that one.
            while (p.subsets > 1 && p.stages <= kLag * p.subsets + p.stages % p.subsets) --p.subsets;
            p.stages -= p.stages % p.subsets;
            if (p.stages <= kLag) continue;
        }
        // the scratch lies at the end, behind all stages where there is room for that
        p.end = p.ring_addr + aligned((size_t)p.stages * stage_bytes) + scratch;
        if (p.end > kWindowEnd) p.end = kWindowEnd;
        p.plane_addr = p.end - scratch;
        p.xchg_addr = p.plane_addr + plane_bytes;
        // The first stages are asked for by one warp while the others prepare the planes and then wait for it: a box to each set and
        // no more (151936x512, sixty stages: all before the planes 9.9 us, twenty 9.2).
        p.early = stages_in(p.plane_addr) < p.stages ? stages_in(p.plane_addr) : p.stages;
        if (p.early > kMaxWarps) p.early = kMaxWarps;
        p.ok = true;
        p.us = tile_us(log, set_warps, p.subsets, per);
        narrow = narrow || log < 2;
        if (!best.ok || p.us < best.us) best = p;
    }
    best.faster = best.ok && (narrow || not_behind_chain(best, tokens, tiles, chunks));
    return best;
}

}  // namespace

bool gemv_tiles_layout(int M, int N, int K, const int *rooms, CallLayout *layout) {
    if (M < 1 || M > kMaxTokens || !gemv_chain_shape_ok(N, K)) return false;
    const TilePlan p = tile_plan(M, N, K, rooms);
    if (!p.ok) return false;
    *layout = {1 << p.split_log, p.subsets, p.stages, ((N + kTileRows - 1) / kTileRows + p.clusters - 1) / p.clusters, p.faster};
    return true;
}

bool try_gemv_tiles(const uint8_t *blocks, const __half *x, void *y, bool y_f32, int M, int N, int K, bool swiglu, void *workspace,
                    cudaStream_t stream, int *status) {
    if (M < 1 || M > kMaxTokens || !gemv_chain_supported(blocks, N, K)) return false;
    const TilePlan p = tile_plan(M, N, K);
    const EncodeTiledFn encode = encode_tiled_fn();
    if (!p.faster || !encode) return false;
    TileParams prm;
    prm.x = x;
    prm.y = y;
    prm.status = static_cast<unsigned *>(workspace);
    prm.N = N;
    prm.chunks = K / kChunkCols;
    prm.tiles = (N + kTileRows - 1) / kTileRows;
    prm.clusters = p.clusters;
    prm.split_log = p.split_log;
    prm.slices = p.slices;
    prm.subsets = p.subsets;
    prm.stages = p.stages;
    prm.pitch = p.pitch;
    prm.early = p.early;
    prm.plane_addr = p.plane_addr;
    prm.xchg_addr = p.xchg_addr;
    prm.sums_addr = p.sums_addr;
    prm.ring_addr = p.ring_addr;
    prm.y_f32 = y_f32 ? 1 : 0;
    prm.swiglu = swiglu ? 1 : 0;
    // A row as 8-byte elements; a box is the 16 rows of a tile and a CTA's K range, at most 16 bytes more (another CTA's, or
    // filled in past the row's end), so that rows lie an odd number of 16-byte units apart.
    CUtensorMap wmap;
    const cuuint64_t row_bytes = (cuuint64_t)prm.chunks * kChunkBytes, dims[2] = {row_bytes / 8, (cuuint64_t)N}, strides[1] = {row_bytes};
    const cuuint32_t box[2] = {(cuuint32_t)p.pitch / 8, kTileRows}, ones[2] = {1, 1};
    const CUresult res = encode(&wmap, CU_TENSOR_MAP_DATA_TYPE_INT64, 2, const_cast<uint8_t *>(blocks), dims, strides, box, ones,
                                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (res != CUDA_SUCCESS) {
        *status = fail(TQ1_ERR_CUDA, "tq1_linear_f16: weight tensor map failed (%d)", (int)res);
        return true;
    }
    const TileKernel kernel = kernel_of(p.split_log > 0, M);
    cudaError_t err = opt_in(g_records[p.split_log > 0][M - 1], reinterpret_cast<const void *>(kernel), kWindowEnd - kWindow);
    if (err != cudaSuccess) {
        *status = cuda_fail(err, "tq1_linear_f16: shared memory opt-in (tiles)");
        return true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(p.clusters << p.split_log));
    // at least a warp to every two groups of activations, which they prepare one after the other
    int warps = p.slices * M * kChunkGroups / 2;
    warps = warps < kMinWarps ? kMinWarps : warps > kMaxWarps ? kMaxWarps : warps;
    if (warps < p.slices * M * p.subsets) warps = p.slices * M * p.subsets;
    cfg.blockDim = dim3((unsigned)(32 * warps));
    cfg.dynamicSmemBytes = p.end - kWindow;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1u << p.split_log;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    const bool captured = stream_captured(stream);
    cfg.numAttrs = !captured || behind_own_kernel(stream) ? 2 : 1;
    err = cudaLaunchKernelEx(&cfg, kernel, wmap, prm);
    if (captured && err == cudaSuccess) note_captured_kernel(stream);
    *status = err == cudaSuccess ? TQ1_OK : cuda_fail(err, "tq1_linear_f16: launch (tiles)");
    return true;
}

}  // namespace tq1
