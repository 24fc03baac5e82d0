// Linear with an FP32 sum per 128-weight group on tcgen05, for the widths and alignments of tq1_gemm_groups.cu (no multiple of
// 512, blocks off the 16-byte grid) where there is enough of it to fill a CTA's pipeline.
//
// The arithmetic is that of tq1_gemm_groups.cu: weights -1, 0, +1 in FP16 times FP16 activations, an accumulator covers 32
// columns (two MMAs: the tensor core truncates when it adds to one), the four of a group are added in FP32, then
// acc = fma(scale, group_sum, acc) with the rounding error carried along (Kahan's summation), so non-finite scales and
// activations come out as in the reference's order (src/bonsai_tq1/reference.py:33-38). 4.0e-8 from the FP64 product (2-norm)
// on 17408x5248, where the mma.sync form has 5.3e-8.
//
// A CTA has a tile of 128 weight rows x up to 64 tokens; a K block is a group.
//   8 warps   decode: two groups of four take K blocks in turn; a lane's row of 28 bytes comes by 4-byte cp.async (rows are
//             4-byte aligned only), goes through the table of PRMT selectors and as 64 registers of FP16 pairs to tensor memory
//   2 warps   issue the MMAs, every second unit each: per K block and unit of 32 tokens eight, on four accumulators
//   16 warps  read the accumulators of a unit (four of them a row, eight tokens each), add, scale, and carry the errors
//   1 warp    fetches the activations by TMA
// Two units' accumulators (256 columns of tensor memory) alternate. Few tiles: a cluster of CTAs splits the groups of a tile and
// adds its sums through distributed shared memory; no workspace is needed.
//
// What bounds it: issue slots (69% used; 6400 instructions per K block of two units, 900 of them the decode, the rest for the
// sums of its 32768 accumulator values) and the round trip of a unit, MMAs - accumulators read and added - slot free again, with
// two slots: 0.64 us a K block of one unit, 1.13 of two (without the sums 0.5 and 0.75; without the decode, or with one of eight
// MMAs, hardly less than with them; one MMA warp, or half as many warps with twice the tokens for the sums, 3% more). Weights
// out of HBM, against the mma.sync forms: 16 / 64 / 700 tokens of 17408x5248 31.8 / 51.8 / 525 us (37.8 / 72 / 735),
// 64 / 129 / 700 of 4099x2176 12.5 / 23.2 / 66.5 (15.7 / 31.3 / 89).
#include <cuda.h>

#include "tq1_common.cuh"
#include "tq1_decode.cuh"

namespace tq1 {

namespace {

constexpr int kTileW = 128, kUnit = 32, kUnits = 2, kTokens = kUnit * kUnits;
constexpr int kRing = 4, kScaleRing = 8, kPackRing = 4;         // a scale outlives its ring stage by two K blocks at most
constexpr int kDecodeWarps = 8, kSumWarps = 16, kMmaWarps = 2;
constexpr int kMmaWarp = kDecodeWarps + kSumWarps, kXWarp = kMmaWarp + kMmaWarps, kThreads = 32 * (kXWarp + 1);
constexpr uint32_t kPackBytes = 32 * kBlockBytes;               // a warp's rows of a K block
constexpr uint32_t kWindow = 1024;                              // shared-window address of dynamic shared memory
constexpr uint32_t kBarAddr = kWindow;
constexpr uint32_t kScaleAddr = kBarAddr + 1024;
constexpr uint32_t kPackAddr = kScaleAddr + kScaleRing * kTileW * 4;
constexpr uint32_t kTableAddr = kPackAddr + kDecodeWarps * kPackRing * kPackBytes;
constexpr uint32_t kStageBytes = kTokens * kGroup * 2;
constexpr uint32_t kBAddr = (kTableAddr + kCodeTableBytes + 1023) / 1024 * 1024;
constexpr uint32_t kRedAddr = kBAddr + kRing * kStageBytes;     // sums from the CTAs of the cluster
constexpr uint32_t kSmemEnd = kRedAddr + kTokens * kTileW * 8;
static_assert(kTableAddr % 256 == 0 && kSmemEnd <= 227 * 1024, "shared memory layout");
constexpr int kAccCols = kUnit * 4;                             // a unit's accumulators
constexpr int kABase = 2 * kAccCols;                            // decoded weights: kRing stages of 64 columns
static_assert(kABase + kRing * 64 <= 512, "tensor memory");

struct GroupParams {
    const uint8_t *blocks;
    void *y;
    unsigned *status;
    int M, N, groups;
    int tiles_m, tiles, clusters, split_log, nt;                // nt: tokens of a tile, the last token tile has what is left
    int y_f32;
};

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ void unpack2(f32x2 v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, bool accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"((uint32_t)accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// Eight columns of two accumulators.
__device__ __forceinline__ void tmem_load8x2(uint32_t a, uint32_t b, f32x2 (&u)[4], f32x2 (&v)[4]) {
    float r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]) : "r"(a) : "memory");
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(r[8]), "=f"(r[9]), "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15]) : "r"(b) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) asm volatile("" : "+f"(r[i]));          // no use before the wait
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        u[i] = pack2(r[2 * i], r[2 * i + 1]);
        v[i] = pack2(r[8 + 2 * i], r[9 + 2 * i]);
    }
}

__global__ void __launch_bounds__(kThreads, 1)
groups_tc_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ GroupParams prm) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const uint32_t window = (uint32_t)__cvta_generic_to_shared(smem);
    const uint32_t base = window - kWindow;                     // zero, or what names this CTA of a cluster
    if ((base & 0x00ffffffu) != 0u) {                           // the fixed window addresses do not hold
        if (threadIdx.x == 0) atomicExch(prm.status, 2u);
        return;
    }
    constexpr int FULL_A = 0, FULL_B = FULL_A + kRing, EMPTY = FULL_B + kRing, ACC_FULL = EMPTY + kRing, ACC_FREE = ACC_FULL + 2;
    auto bar = [base](int i) { return base + kBarAddr + 8u * (uint32_t)i; };
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(smem + (kBarAddr - kWindow) + 1008);
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int split_log = prm.split_log, split = 1 << split_log, rank = blockIdx.x & (split - 1), cluster = blockIdx.x >> split_log;
    const int g0 = prm.groups * rank >> split_log, blocks_k = (prm.groups * (rank + 1) >> split_log) - g0;

    if (tid == 0) {
        for (int i = 0; i < kRing; ++i) {
            mbar_init(bar(FULL_A + i), 4);
            mbar_init(bar(FULL_B + i), 1);
            mbar_init(bar(EMPTY + i), 2);                       // two units' MMAs, or those of one twice
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar(ACC_FULL + i), 2);                    // the MMAs, and their thread, which has seen the scales written
            mbar_init(bar(ACC_FREE + i), kSumWarps);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(base + kBarAddr + 1008) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (warp == kXWarp && lane == 0) asm volatile("prefetch.tensormap [%0];" ::"l"(&xmap) : "memory");
    fill_code_table(smem + (kTableAddr - kWindow), warp, kThreads / 32, lane);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (split > 1) {                                            // the CTAs of a cluster write into each other's memory
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        __syncthreads();
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    allow_next_grid();                                          // its CTAs have no room beside these
    grid_dependency_wait();

    bool dead = false;
    auto token0 = [&](int tile) { return tile % prm.tiles_m * prm.nt; };
    auto units_of = [&](int m0) { return (min(prm.nt, prm.M - m0) + kUnit - 1) / kUnit; };
    auto unit_tokens = [&](int m0, int u) { return (min(kUnit, min(prm.nt, prm.M - m0) - u * kUnit) + 15) / 16 * 16; };

    if (warp == kXWarp) {
        // ------------------------------------------------------------------ activations
        if (elect_one()) {
            uint32_t i = 0;
            const uint32_t bytes = (uint32_t)prm.nt * 256u;
            for (int tile = cluster; tile < prm.tiles && !dead; tile += prm.clusters) {
                const int m0 = token0(tile);
                for (int kb = 0; kb < blocks_k; ++kb, ++i) {
                    const uint32_t stage = i % kRing;
                    mbar_wait(bar(EMPTY + (int)stage), (i / kRing & 1u) ^ 1u, prm.status, dead);
                    if (dead) break;
                    mbar_expect_tx(bar(FULL_B + (int)stage), bytes);
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                                     ::"r"(base + kBAddr + stage * kStageBytes + (uint32_t)h * (bytes / 2)), "l"(&xmap),
                                       "r"((g0 + kb) * kGroup + 64 * h), "r"(m0), "r"(bar(FULL_B + (int)stage)) : "memory");
                }
            }
        }
    } else if (warp >= kMmaWarp) {
        // ------------------------------------------------------------------ MMAs: every second unit, and one of the two slots
        if (elect_one()) {
            const uint32_t slot = (uint32_t)(warp - kMmaWarp);
            uint32_t i = 0, unit = 0, last_bar = 0, last_phase = 0;
            for (int tile = cluster; tile < prm.tiles && !dead; tile += prm.clusters) {
                const int m0 = token0(tile), units = units_of(m0);
                for (int kb = 0; kb < blocks_k; ++kb, ++i, unit += (uint32_t)units) {
                    const int u = (int)((slot ^ unit) & 1u);    // this warp's unit of the block
                    if (u >= units) continue;
                    const uint32_t stage = i % kRing, phase = i / kRing & 1u;
                    const uint32_t idesc = (1u << 4) | ((uint32_t)(unit_tokens(m0, u) >> 3) << 17) | ((uint32_t)(kTileW >> 4) << 24);
                    const uint32_t a_tmem = tmem_base + (uint32_t)kABase + stage * 64u;
                    const uint32_t b_lo = base + kBAddr + stage * kStageBytes + (uint32_t)u * (kUnit * 128u);
                    const uint64_t lo = umma_desc(b_lo), hi = umma_desc(b_lo + (uint32_t)prm.nt * 128u);
                    mbar_wait(bar(ACC_FREE + (int)slot), ((unit + (uint32_t)u) >> 1 & 1u) ^ 1u, prm.status, dead);
                    mbar_wait(bar(FULL_B + (int)stage), phase, prm.status, dead);
                    mbar_wait(bar(FULL_A + (int)stage), phase, prm.status, dead);
                    if (dead) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (int j = 0; j < 8; ++j)                 // two K = 16 steps per accumulator
                        umma_f16_ts(tmem_base + slot * kAccCols + (uint32_t)(j >> 1) * kUnit, a_tmem + 8u * j,
                                    (j < 4 ? lo : hi) + 2u * (j & 3), idesc, j & 1);
                    umma_commit(bar(ACC_FULL + (int)slot));
                    umma_commit(bar(EMPTY + (int)stage));
                    if (units == 1) umma_commit(bar(EMPTY + (int)stage));
                    mbar_arrive(bar(ACC_FULL + (int)slot));
                    last_bar = bar(EMPTY + (int)stage);
                    last_phase = phase;
                }
            }
            // Nothing of this warp's commits arrives after the last of them, which this phase has to have. With one unit per
            // block that is not the last block's: the warps take turns, and commits of different threads come in any order.
            if (last_bar) mbar_wait(last_bar, last_phase, prm.status, dead);
        }
    } else if (warp < kDecodeWarps) {
        // ------------------------------------------------------------------ decode
        const int group = warp >> 2, quad = warp & 3;
        const uint32_t tmem_lane = tmem_base + ((uint32_t)(quad * 32) << 16);
        const uint32_t even_entry = base | ((uint32_t)(lane & 15) * 8u), odd_entry = even_entry | 128u;
        const uint32_t pack = base + kPackAddr + (uint32_t)(warp * kPackRing) * kPackBytes;
        const long long row_bytes = (long long)prm.groups * kBlockBytes;
        // The warp's 32 rows of a K block are 224 words; a lane copies word lane + 32 j. K blocks are numbered over all tiles
        // of the CTA, this warp has every second one.
        auto normalise = [&](int &tile, int &kb) {
            while (kb >= blocks_k && tile < prm.tiles) { kb -= blocks_k; tile += prm.clusters; }
        };
        int p_tile = cluster, p_kb = group, p_slot = 0;
        normalise(p_tile, p_kb);
        auto request = [&]() {
            if (p_tile < prm.tiles) {
                const int n0 = p_tile / prm.tiles_m * kTileW + quad * 32;
                const uint8_t *src = prm.blocks + (long long)n0 * row_bytes + (long long)(g0 + p_kb) * kBlockBytes;
#pragma unroll
                for (int j = 0; j < 7; ++j) {
                    const int w = lane + 32 * j, row = w / 7, word = w - 7 * row;
                    const bool in = n0 + row < prm.N;           // rows past the end: zeros
                    const uint8_t *from = in ? src + row * row_bytes + word * 4 : prm.blocks;
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;"
                                 ::"r"(pack + (uint32_t)p_slot * kPackBytes + (uint32_t)w * 4u), "l"(from), "r"(in ? 4 : 0) : "memory");
                }
                p_kb += 2;
                normalise(p_tile, p_kb);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            if (++p_slot == kPackRing) p_slot = 0;
        };
#pragma unroll
        for (int s = 0; s < kPackRing - 1; ++s) request();
        uint32_t i = (uint32_t)group;
        int tile = cluster, kb = group, slot = 0;
        normalise(tile, kb);
        for (; tile < prm.tiles; kb += 2, i += 2, normalise(tile, kb)) {
            request();
            asm volatile("cp.async.wait_group %0;" ::"n"(kPackRing - 1) : "memory");
            __syncwarp();
            uint32_t w[7];
            const uint32_t src = pack + (uint32_t)slot * kPackBytes + (uint32_t)lane * kBlockBytes;
#pragma unroll
            for (int k = 0; k < 7; ++k) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w[k]) : "r"(src + 4u * k) : "memory");
            __syncwarp();                                       // the buffer may be requested again
            if (++slot == kPackRing) slot = 0;
            const RowDecoder<kTableAddr> row{w, 0x00bc3c00u, even_entry, odd_entry};        // FP16 weights -1, 0, +1
            const uint32_t stage = i % kRing;
            const uint32_t a_addr = tmem_lane + (uint32_t)kABase + stage * 64u;
            uint32_t v[32], m0w, m1w;                           // byte 12 belongs to both halves
#pragma unroll
            for (int a = 0; a < 6; ++a) row.two_bytes(2 * a, v + 5 * a);
            row.lookup(12, m0w, m1w);
            v[30] = row.pick(m0w);
            v[31] = row.pick(m1w);
            mbar_wait(bar(EMPTY + (int)stage), (i / kRing & 1u) ^ 1u, prm.status, dead);
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            tmem_store32(a_addr, v);
            {
                uint32_t f0, f1, e0, e1;
                row.lookup(13, f0, f1);
                v[0] = row.pick(prmt(m0w, f0, 0x0062));
                v[1] = row.pick(f0);
                v[2] = row.pick(f1);
#pragma unroll
                for (int a = 0; a < 5; ++a) row.two_bytes(14 + 2 * a, v + 3 + 5 * a);
                row.lookup(24, e0, e1);
                row.lookup(25, f0, f1);                         // the tail byte's three trits
                v[28] = row.pick(e0);
                v[29] = row.pick(e1);
                v[30] = row.pick(prmt(e0, f0, 0x0062));
                v[31] = row.pick(f0);
            }
            tmem_store32(a_addr + 32u, v);
            reinterpret_cast<float *>(smem + (kScaleAddr - kWindow))[i % kScaleRing * kTileW + quad * 32 + lane] =
                __half2float(__ushort_as_half((unsigned short)(w[0] & 0xffffu)));
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(FULL_A + (int)stage));
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
        // ------------------------------------------------------------------ sums and results
        const int part = (warp - kDecodeWarps) >> 2, quad = warp & 3, row = quad * 32 + lane;        // part: which tokens of a unit
        const uint32_t tmem_lane = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(8 * part);
        const float *scales = reinterpret_cast<const float *>(smem + (kScaleAddr - kWindow)) + row;
        const f32x2 minus = pack2(-1.0f, -1.0f);
        uint32_t i = 0, unit = 0;
        for (int tile = cluster; tile < prm.tiles; tile += prm.clusters) {
            const int m0 = token0(tile), units = units_of(m0);
            f32x2 acc[kUnits][4], carry[kUnits][4];             // sums, and what their roundings have lost
#pragma unroll
            for (int u = 0; u < kUnits; ++u)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[u][c] = carry[u][c] = 0ull;
            for (int kb = 0; kb < blocks_k; ++kb, ++i) {
                f32x2 scale = 0ull;
#pragma unroll
                for (int u = 0; u < kUnits; ++u) {
                    if (u >= units) continue;
                    const uint32_t slot = unit & 1u;
                    mbar_wait(bar(ACC_FULL + (int)slot), unit >> 1 & 1u, prm.status, dead);
                    __syncwarp();
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (u == 0) {
                        const float s = scales[i % kScaleRing * kTileW];
                        scale = pack2(s, s);
                    }
                    if (8 * part < unit_tokens(m0, u)) {
                        const uint32_t at = tmem_lane + slot * kAccCols;
                        f32x2 finite = 0ull, a[4], b[4], c[4], d[4];
                        tmem_load8x2(at, at + kUnit, a, b);
#pragma unroll
                        for (int e = 0; e < 4; ++e) a[e] = add2(a[e], b[e]);
                        tmem_load8x2(at + 2 * kUnit, at + 3 * kUnit, c, d);
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const f32x2 sum = add2(a[e], add2(c[e], d[e]));
                            const f32x2 value = fma2(scale, sum, carry[u][e]), next = add2(acc[u][e], value);
                            carry[u][e] = fma2(minus, fma2(minus, acc[u][e], next), value);      // value - (next - acc)
                            acc[u][e] = next;
                            finite = fma2(next, 0ull, finite);
                        }
                        float f0, f1;
                        unpack2(finite, f0, f1);
                        if (!(f0 + f1 == 0.0f)) {               // an infinite sum stays what it is: nothing is carried along with it
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                float x0, x1;
                                unpack2(carry[u][e], x0, x1);
                                carry[u][e] = pack2(fabsf(x0) <= 3.4028235e38f ? x0 : 0.0f, fabsf(x1) <= 3.4028235e38f ? x1 : 0.0f);
                            }
                        }
                    }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar(ACC_FREE + (int)slot));
                    ++unit;
                }
            }
            const int n = tile / prm.tiles_m * kTileW + row, tokens = min(prm.nt, prm.M - m0);
#pragma unroll
            for (int u = 0; u < kUnits; ++u)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    float r[2], lost[2];
                    unpack2(acc[u][c], r[0], r[1]);
                    unpack2(carry[u][c], lost[0], lost[1]);
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int t = u * kUnit + 8 * part + 2 * c + e;
                        if (t >= tokens) continue;
                        if (split_log > 0) {                    // with its error to the CTA of the cluster that has the token
                            uint32_t dst;
                            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst)
                                         : "r"(base + kRedAddr + 8u * (uint32_t)(((t & ~(split - 1)) + rank) * kTileW + row)), "r"(t & (split - 1)));
                            asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(dst), "f"(r[e]), "f"(lost[e]) : "memory");
                        } else if (n < prm.N) {
                            const size_t o = (size_t)(m0 + t) * prm.N + n;
                            if (!TQ1_IN_BOUNDS(o, (size_t)prm.M * prm.N, 70u)) continue;
                            if (prm.y_f32) static_cast<float *>(prm.y)[o] = r[e];
                            else static_cast<__half *>(prm.y)[o] = __float2half_rn(r[e]);
                        }
                    }
                }
        }
    }

    __syncwarp();
    if (dead)                                                   // a wait ran out: give the copies still in flight time to land
        for (int i = 0; i < 64; ++i) __nanosleep(20000);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (split > 1) {
        // a cluster has one tile; this CTA adds the parts of every split-th token in the order of the columns
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        const float2 *red = reinterpret_cast<const float2 *>(smem + (kRedAddr - kWindow));
        const int m0 = token0(cluster), tokens = min(prm.nt, prm.M - m0), n0 = cluster / prm.tiles_m * kTileW;
        for (int j = tid; (j / kTileW << split_log) + rank < tokens; j += kThreads) {
            const int t = (j / kTileW << split_log) + rank, r = j % kTileW;
            if (n0 + r >= prm.N) continue;
            double v = 0.0;                                     // one rounding for the sum of the parts
            for (int c = 0; c < split; ++c) {
                const float2 p = red[((t & ~(split - 1)) + c) * kTileW + r];
                v += (double)p.x + (double)p.y;
            }
            const size_t o = (size_t)(m0 + t) * prm.N + n0 + r;
            if (!TQ1_IN_BOUNDS(o, (size_t)prm.M * prm.N, 70u)) continue;
            if (prm.y_f32) static_cast<float *>(prm.y)[o] = (float)v;
            else static_cast<__half *>(prm.y)[o] = __float2half_rn((float)v);
        }
        __syncwarp();
    } else {
        __syncthreads();
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
    }
}

// ---- host ---------------------------------------------------------------------------------------------------------
KernelRecord g_record;
const void *const kKernel = reinterpret_cast<const void *>(groups_tc_kernel);
int clusters_at_once(int split_log) { return tq1::clusters_at_once(g_record, kKernel, kThreads, kSmemEnd - kWindow, 1 << split_log); }

struct GroupPlan { int nt, tiles_m, tiles, clusters, split; float us; };

// Token tiles of equal length, and as many CTAs to a tile as leave every cluster one tile and each of its CTAs four groups.
GroupPlan group_plan(int M, int N, int groups) {
    GroupPlan p;
    p.tiles_m = (M + kTokens - 1) / kTokens;
    p.nt = ((M + p.tiles_m - 1) / p.tiles_m + 15) / 16 * 16;
    p.tiles_m = (M + p.nt - 1) / p.nt;
    p.tiles = (N + kTileW - 1) / kTileW * p.tiles_m;
    int split_log = 0;
    while (split_log < 3 && p.tiles <= clusters_at_once(split_log + 1) && groups >= 8 << split_log) ++split_log;
    p.split = 1 << split_log;
    const int room = clusters_at_once(split_log);
    p.clusters = p.tiles < room ? p.tiles : room;
    const int tiles = (p.tiles + p.clusters - 1) / p.clusters, blocks = tiles * ((groups + p.split - 1) / p.split);
    p.us = p.nt <= kUnit ? 4.37f + 1.41f * (float)tiles + 0.643f * (float)blocks + (p.split > 1 ? 1.1f : 0.0f) +
                               55.5e-9f * (float)N * (float)(groups * kGroup)
                         : 6.5f + 1.13f * (float)blocks;
    return p;
}

}  // namespace

float gemm_groups_tc_us(int M, int N, int K) { return group_plan(M, N, K / kGroup).us; }

int launch_gemm_groups_tc(const uint8_t *blocks, const __half *x, void *y, bool y_f32, int M, int N, int K, unsigned *status,
                          cudaStream_t stream) {
    const GroupPlan p = group_plan(M, N, K / kGroup);
    GroupParams prm;
    prm.blocks = blocks;
    prm.y = y;
    prm.status = status;
    prm.M = M;
    prm.N = N;
    prm.groups = K / kGroup;
    prm.tiles_m = p.tiles_m;
    prm.tiles = p.tiles;
    prm.clusters = p.clusters;
    prm.split_log = p.split == 1 ? 0 : p.split == 2 ? 1 : p.split == 4 ? 2 : 3;
    prm.nt = p.nt;
    prm.y_f32 = y_f32 ? 1 : 0;
    const EncodeTiledFn encode = encode_tiled_fn();
    if (!encode) return fail(TQ1_ERR_CUDA, "tq1_linear_f16: cuTensorMapEncodeTiled is unavailable");
    CUtensorMap xmap;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)M}, strides[1] = {(cuuint64_t)K * sizeof(__half)};
    const cuuint32_t box[2] = {64, (cuuint32_t)p.nt}, ones[2] = {1, 1};
    const CUresult res = encode(&xmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half *>(x), dims, strides, box, ones,
                                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (res != CUDA_SUCCESS) return fail(TQ1_ERR_CUDA, "tq1_linear_f16: activation tensor map failed (%d)", (int)res);
    cudaError_t err = opt_in(g_record, kKernel, kSmemEnd - kWindow);
    if (err != cudaSuccess) return cuda_fail(err, "tq1_linear_f16: shared memory opt-in (group sums)");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(p.clusters * p.split));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemEnd - kWindow;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)p.split;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    const bool captured = stream_captured(stream);
    cfg.numAttrs = !captured || behind_own_kernel(stream) ? 2 : 1;
    err = cudaLaunchKernelEx(&cfg, groups_tc_kernel, xmap, prm);
    if (captured && err == cudaSuccess) note_captured_kernel(stream);
    return err == cudaSuccess ? TQ1_OK : cuda_fail(err, "tq1_linear_f16: launch (group sums)");
}

}  // namespace tq1
