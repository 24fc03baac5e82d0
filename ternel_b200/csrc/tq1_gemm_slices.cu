// Linear of a few activation rows (3 to 16) for widths that are multiples of 512: decoded weights are the A operand of
// mma.sync.m16n8k16, straight out of registers.
//
// The tcgen05 kernel needs 128 weight rows, tensor memory and a K split over CTAs with partial tiles through L2 for such calls:
// about 7 us before and after the weights, and 311 instructions per 32 rows x 128 columns. Here decoded weights never leave the
// registers of the warp that decoded them, and a row's sum never leaves the CTA (or its cluster).
//
//   slice     a K range of one warp: a 512-column chunk for up to eight tokens, half of one for sixteen (64 registers of
//             activations either way). Lane (g, q) of a warp takes rows g and g + 8 of a 16-row tile and, in group q of the
//             chunk, 64 consecutive columns at a time. The contraction may take the columns in any order as long as both operands
//             agree, so the lane's consecutive weight pairs are the A registers of consecutive MMAs (four columns of each
//             group of the chunk) and its 128 bytes of activations the B registers.
//   warp      keeps the activations of its slice in registers and streams row tiles past it
//   CTA       `slices` warps cover a K range, `subsets` such sets of warps take turns on the row tiles; one more warp fetches
//             the tiles, 16 rows of the CTA's K range by one TMA box, into a ring (a bulk copy per row, from 16 lanes, took 240
//             clocks per row to issue). Rows lie an odd number of 16-byte units apart: no bank conflicts between them.
//   cluster   1, 2, 4 or 8 CTAs split K between them and add their sums through distributed shared memory
//
// The slices' sums of a tile meet in shared memory; the set's warps take turns with adding them, two tiles later, in a fixed
// order (a warp that did nothing else needed 2500 clocks a tile beside twenty that decode, and set the pace).
//
// As in the tcgen05 kernel the group scale is folded into the FP16 weight, which is exact, and a code byte becomes PRMT
// selectors by one lookup in a table with sixteen copies of an entry (src/ternel_mlx/kernels.py:435-440 of the reference
// folds the scale the same way). A tensor-core accumulator covers 64 columns, everything above is FP32 additions: 1.3e-7 from
// the FP64 product (2-norm) at every width, where the tcgen05 kernel has 1.8e-7 (512 columns) to 7.5e-7 (17408).
//
// What bounds it: few rows, the chain launch - activations - words - lookups - MMAs - sums; many rows, the instructions of the
// decode with ten warps to hide their latencies (40% of issue slots, ALU 40%, shared memory 40%). 8 tokens, weights out of HBM,
// against the tcgen05 kernel: 1024x5120 3.7 us (10.2), 4096x4096 5.5 (10.3), 5120x5120 7.9 (11.0), 17408x5120 14.5 (17.6),
// 34816x5120 23.8 (26.3), 5120x17408 18.3 (18.9). Twenty warps with half a chunk each were as fast (322 instructions instead of
// 253 per 16 rows x 256 columns); so were four warps for the sums, and fetching a tile's words before the sums before it.
#include <cuda.h>

#include <type_traits>

#include "tq1_common.cuh"
#include "tq1_decode.cuh"

namespace tq1 {

namespace {

constexpr int kTileRows = 16;
constexpr int kChunkBytes = 4 * kBlockBytes;                    // a row's bytes of a 512-column chunk
constexpr int kChain = 4;                                       // MMAs (of 16 columns) under one accumulator

constexpr uint32_t kWindow = 1024;                              // shared-window address of dynamic shared memory
constexpr uint32_t kTableAddr = kWindow;                        // 256 entries of 256 bytes
constexpr uint32_t kBarAddr = kTableAddr + kCodeTableBytes;
constexpr uint32_t kBarBytes = 2048;
constexpr uint32_t kDataAddr = kBarAddr + kBarBytes;            // activations and later partial sums, sums (split K), ring
constexpr uint32_t kXBytes = 4096;                              // activations: half a chunk, eight tokens
constexpr uint32_t kWindowEnd = 227 * 1024;
constexpr int kTokenPitch = 20;                                 // floats from one token's 16 rows to the next: no conflicts
constexpr int kTokenTile = 8 * kTokenPitch;                     // floats of eight tokens
__host__ __device__ constexpr int part_floats(int nt) { return nt * kTokenTile + 8; }      // one slice's sums of a row tile
constexpr int kLag = 2;                                         // a tile is added up while the second one after it is decoded
constexpr int kBufs = 2 * kLag;                                 // row tiles whose sums are kept, per set of warps
constexpr int kMaxStages = 24;

// Warps that decode: 12 warps leave each 168 registers.
constexpr int kMaxSlices = 11;
constexpr int kMaxOwn = 96;                                     // row tiles that a CTA of a cluster adds up
static_assert(8 * (2 * kMaxStages + kBufs * kMaxSlices + kMaxSlices + kMaxOwn) <= kBarBytes, "barrier area");
__host__ __device__ constexpr int slice_halves(int nt) { return nt == 1 ? 2 : 1; }          // 64 registers of activations
constexpr int kExtraWarps = 1;
// Fewer warps than this would be long at filling the table (two of them: 1.1 us more than six; 8 tokens of 2048x512 6.5 us apart
// from other calls, 5.4 with six, 5.2 with nine). Six leave half of the registers to the next call's CTAs: in a row 3.8, 3.1 and 3.9.
constexpr int kFillWarps = 6;

struct SliceParams {
    void *y;
    unsigned *status;
    int M, N, chunks;
    int tiles, clusters;                                        // row tiles, clusters of the grid
    int split_log, slices, subsets, workers;                    // the grid's clusters have 2^split_log CTAs; workers: slices * subsets
    int stages, pitch;                                          // ring stages, bytes from row to row
    int x_bufs;                                                 // 4 KiB pieces of activations that a slice has room for at a time
    uint32_t sums_addr, ring_addr;
    int y_f32, swiglu;
    int wide_y;                                                 // four results of a token may be stored at a time
};

template <int OFFSET>
__device__ __forceinline__ uint32_t lds(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(addr), "n"(OFFSET) : "memory");
    return v;
}
__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1, bool first) {
    if (first)
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
            : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
    else
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The products of one row tile and half a chunk: added to sum[token tile][..] (rows g and g + 8, tokens 2q and 2q + 1).
using Decoder = RowDecoder<kTableAddr>;

// START: these are the first products of sum.
template <int NT, int HALF, bool START>
__device__ __forceinline__ void half_slice(const Decoder &lo, const Decoder &hi, const uint32_t (&b)[NT][32],
                                           float (&sum)[NT][4]) {
    uint32_t va[32], vb[32];
    float d[NT][4];
    auto multiply = [&](int i) {                                // the MMA of registers 2i and 2i + 1
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            mma16816(d[t], va[2 * i], vb[2 * i], va[2 * i + 1], vb[2 * i + 1], b[t][2 * i], b[t][2 * i + 1], i % kChain == 0);
            if (i % kChain == kChain - 1) {
#pragma unroll
                for (int e = 0; e < 4; ++e) sum[t][e] = START && i == kChain - 1 ? d[t][e] : sum[t][e] + d[t][e];
            }
        }
    };
    if (HALF == 0) {
#pragma unroll
        for (int a = 0; a < 6; ++a) {
            lo.two_bytes(2 * a, va + 5 * a);
            hi.two_bytes(2 * a, vb + 5 * a);
#pragma unroll
            for (int i = 0; i < 15; ++i)
                if (2 * i + 1 >= 5 * a && 2 * i + 1 < 5 * a + 5) multiply(i);
        }
        uint32_t e0, e1;                                        // the first four trits of byte 12
        lo.lookup(12, e0, e1);
        va[30] = lo.pick(e0);
        va[31] = lo.pick(e1);
        hi.lookup(12, e0, e1);
        vb[30] = hi.pick(e0);
        vb[31] = hi.pick(e1);
        multiply(15);
    } else {
        auto first = [](const Decoder &r, uint32_t *v) {     // the last trit of byte 12, and byte 13
            uint32_t e0, e1, f0, f1;
            r.lookup(12, e0, e1);
            r.lookup(13, f0, f1);
            v[0] = r.pick(prmt(e0, f0, 0x0062));
            v[1] = r.pick(f0);
            v[2] = r.pick(f1);
        };
        first(lo, va);
        first(hi, vb);
        multiply(0);
#pragma unroll
        for (int a = 0; a < 5; ++a) {
            lo.two_bytes(14 + 2 * a, va + 3 + 5 * a);
            hi.two_bytes(14 + 2 * a, vb + 3 + 5 * a);
#pragma unroll
            for (int i = 1; i < 14; ++i)
                if (2 * i + 1 >= 3 + 5 * a && 2 * i + 1 < 8 + 5 * a) multiply(i);
        }
        auto last = [](const Decoder &r, uint32_t *v) {      // byte 24 and the tail byte's three trits
            uint32_t e0, e1, f0, f1;
            r.lookup(24, e0, e1);
            r.lookup(25, f0, f1);
            v[0] = r.pick(e0);
            v[1] = r.pick(e1);
            v[2] = r.pick(prmt(e0, f0, 0x0062));
            v[3] = r.pick(f0);
        };
        last(lo, va + 28);
        last(hi, vb + 28);
        multiply(14);
        multiply(15);
    }
}

// Four neighbouring rows from n of token m: results.
__device__ __forceinline__ void store_rows(const SliceParams &prm, int n, int m, float4 v) {
    if (m >= prm.M || n >= prm.N) return;
    if (prm.swiglu) {                                           // (gate, up) row pairs: silu(gate) * up
        const size_t o = (size_t)m * (prm.N >> 1) + (n >> 1);
        const float r[2] = {swiglu_f32(v.x, v.y), swiglu_f32(v.z, v.w)};
#pragma unroll
        for (int e = 0; e < 2; ++e)
            if (n + 2 * e < prm.N && TQ1_IN_BOUNDS(o + e, (size_t)prm.M * (prm.N >> 1), 80u)) {
                if (prm.y_f32) static_cast<float *>(prm.y)[o + e] = r[e];
                else static_cast<__half *>(prm.y)[o + e] = __float2half_rn(r[e]);
            }
        return;
    }
    const size_t o = (size_t)m * prm.N + n;
    if (!TQ1_IN_BOUNDS(o + min(4, prm.N - n) - 1, (size_t)prm.M * prm.N, 80u)) return;
    if (prm.wide_y) {
        if (prm.y_f32) {
            *reinterpret_cast<float4 *>(static_cast<float *>(prm.y) + o) = v;
        } else {
            const __half2 lo = __floats2half2_rn(v.x, v.y), hi = __floats2half2_rn(v.z, v.w);
            *reinterpret_cast<uint2 *>(static_cast<__half *>(prm.y) + o) =
                make_uint2(reinterpret_cast<const uint32_t &>(lo), reinterpret_cast<const uint32_t &>(hi));
        }
        return;
    }
    const float r[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int e = 0; e < 4; ++e)
        if (n + e < prm.N) {
            if (prm.y_f32) static_cast<float *>(prm.y)[o + e] = r[e];
            else static_cast<__half *>(prm.y)[o + e] = __float2half_rn(r[e]);
        }
}

__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
// Sum over the four lanes that differ in bits 3 and 4 of their number, in every one of them.
__device__ __forceinline__ float4 join4(float4 v) {
#pragma unroll
    for (int step = 8; step <= 16; step *= 2)
        v = add4(v, make_float4(__shfl_xor_sync(0xffffffffu, v.x, step), __shfl_xor_sync(0xffffffffu, v.y, step),
                                __shfl_xor_sync(0xffffffffu, v.z, step), __shfl_xor_sync(0xffffffffu, v.w, step)));
    return v;
}

template <int NT>
__global__ void __launch_bounds__(32 * (kMaxSlices + kExtraWarps), 1)
slices_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap,
              const __grid_constant__ SliceParams prm) {
    constexpr int kPart = part_floats(NT), HS = slice_halves(NT);
    extern __shared__ __align__(1024) unsigned char smem[];
    const uint32_t window = (uint32_t)__cvta_generic_to_shared(smem);
    const uint32_t base = window - kWindow;                     // zero, or what names this CTA of a cluster
    if ((base & 0x00ffffffu) != 0u) {                           // the fixed window addresses do not hold
        if (threadIdx.x == 0) atomicExch(prm.status, 2u);
        return;
    }
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int warps = blockDim.x >> 5, workers = prm.workers;
    const int split_log = prm.split_log, split = 1 << split_log, rank = blockIdx.x & (split - 1), cluster = blockIdx.x >> split_log;
    // this CTA's slices and row tiles
    const int all = 2 * prm.chunks / HS, slice_lo = all * rank >> split_log, n_slices = (all * (rank + 1) >> split_log) - slice_lo;
    const int chunk_lo = slice_lo * HS >> 1;
    const int tile_lo = (int)((long long)cluster * prm.tiles / prm.clusters);
    const int n_tiles = (int)((long long)(cluster + 1) * prm.tiles / prm.clusters) - tile_lo;
    const uint32_t stage_bytes = (uint32_t)(kTileRows * prm.pitch);
    auto full_bar = [&](int s) { return base + kBarAddr + 8u * (uint32_t)s; };
    auto empty_bar = [&](int s) { return base + kBarAddr + 8u * (uint32_t)(kMaxStages + s); };
    auto sum_bar = [&](int s) { return base + kBarAddr + 8u * (uint32_t)(2 * kMaxStages + s); };
    // clusters: one for each row tile that this CTA adds up, behind those of the slices' activations
    auto tile_bar = [&](int s) { return base + kBarAddr + 8u * (uint32_t)(2 * kMaxStages + kBufs * prm.subsets + kMaxSlices + s); };
    const int own_tiles = (n_tiles - rank + split - 1) >> split_log;
    auto x_bar = [&](int s) { return base + kBarAddr + 8u * (uint32_t)(2 * kMaxStages + kBufs * prm.subsets + s); };

    // ---- set-up that depends on no earlier kernel ---------------------------------------------------------------
    if (tid == 0) {
        for (int s = 0; s < prm.stages; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), (uint32_t)n_slices);
        }
        for (int s = 0; s < kBufs * prm.subsets; ++s) {
            mbar_init(sum_bar(s), (uint32_t)n_slices);
        }
        for (int s = 0; s < n_slices; ++s) mbar_init(x_bar(s), 1);
        if (split > 1)
            for (int s = 0; s < own_tiles; ++s) mbar_init(tile_bar(s), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (tid == 0 && split > 1)                                  // the sums of all of the cluster's CTAs
        for (int s = 0; s < own_tiles; ++s) mbar_expect_tx(tile_bar(s), (uint32_t)(split * NT * 8 * kTileRows * 4));
    const int word_x = chunk_lo * (kChunkBytes / 8);            // the map's elements are 8 bytes
    if (tid == 32) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&wmap) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&xmap) : "memory");
    }
    if (warp == workers && elect_one())                         // the first tiles: into L2 (a hint, whatever they hold by now)
        for (int i = 0; i < min(prm.stages, n_tiles); ++i)
            asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];"
                         ::"l"(&wmap), "r"(word_x), "r"((tile_lo + i) * kTileRows) : "memory");
    fill_code_table(smem + (kTableAddr - kWindow), warp, warps, lane);
    if (split > 1) {                                            // the CTAs of a cluster write into each other's memory
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        __syncthreads();
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");

    bool dead = false;
    if (warp == workers) {
        // ------------------------------------------------------------------ fetch
        if (elect_one()) {
            int stage = 0;
            uint32_t phase = 1;
            for (int i = 0; i < n_tiles; ++i) {
                mbar_wait(empty_bar(stage), phase, prm.status, dead);
                if (dead) break;
                mbar_expect_tx(full_bar(stage), stage_bytes);
                asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                             ::"r"(base + prm.ring_addr + (uint32_t)stage * stage_bytes), "l"(&wmap), "r"(word_x),
                               "r"((tile_lo + i) * kTileRows), "r"(full_bar(stage)) : "memory");
                if (++stage == prm.stages) { stage = 0; phase ^= 1u; }
            }
        }
        __syncwarp();
    } else if (warp < workers) {
        // ------------------------------------------------------------------ decode and multiply
        const int subset = warp / prm.slices, slice = warp - subset * prm.slices, g = lane >> 2, q = lane & 3;
        const int half0 = (slice_lo + slice) * HS, chunk = half0 >> 1;
        // This lane's 64 columns of tokens 8t + g: TMA brings the warp's 32 pieces of 128 bytes (16-byte loads from global
        // memory touch 32 lines each, which took the warps of a CTA 2.7 us).
        uint32_t b[HS][NT][32];
        const uint32_t x_addr = base + kDataAddr + (uint32_t)(slice * prm.x_bufs) * kXBytes;
        if (slice < n_slices) {
#pragma unroll
            for (int j = 0; j < HS * NT; ++j) {                 // a half of eight tokens each
                if (j % prm.x_bufs == 0) {                      // the next x_bufs of them; one set of warps asks for all
                    if (warp == slice && elect_one()) {
                        mbar_expect_tx(x_bar(slice), (uint32_t)prm.x_bufs * kXBytes);
                        for (int u = j; u < j + prm.x_bufs; ++u)
                            asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes "
                                         "[%0], [%1, {%2, %3, %4, %5}], [%6];"
                                         ::"r"(x_addr + (uint32_t)(u - j) * kXBytes), "l"(&xmap), "r"(0),
                                           "r"(HS == 2 ? u : half0 & 1), "r"(4 * chunk), "r"(HS == 2 ? 0 : 8 * u),
                                           "r"(x_bar(slice)) : "memory");
                    }
                    __syncwarp();
                    mbar_wait(x_bar(slice), (uint32_t)(j / prm.x_bufs) & 1u, prm.status, dead);
                }
                const uint32_t src = x_addr + (uint32_t)(j % prm.x_bufs) * kXBytes + (uint32_t)lane * 128u;
                uint32_t (&to)[32] = b[HS == 2 ? j : 0][HS == 2 ? 0 : j];
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                                 : "=r"(to[4 * i]), "=r"(to[4 * i + 1]), "=r"(to[4 * i + 2]), "=r"(to[4 * i + 3])
                                 : "r"(src + (uint32_t)((i ^ (lane & 7)) << 4)) : "memory");
                __syncwarp();
            }
        }
        asm volatile("bar.sync 1, %0;" ::"r"(workers * 32) : "memory");      // the partial sums take the activations' place
        if (slice < n_slices) {
            const uint32_t even_entry = base | ((uint32_t)(lane & 15) * 8u), odd_entry = even_entry | 128u;
            const uint32_t lane_src = base + prm.ring_addr + (uint32_t)(g * prm.pitch + (chunk - chunk_lo) * kChunkBytes + q * kBlockBytes);
            float *parts = reinterpret_cast<float *>(smem + (kDataAddr - kWindow)) + subset * (kBufs * prm.slices * kPart);
            float *lane_dst = parts + slice * kPart + 2 * q * kTokenPitch + g;
            const uint32_t row8 = 8u * (uint32_t)prm.pitch, own_sum_bar = sum_bar(kBufs * subset);
            // Adding the slices of the set's k-th row tile is 4 NT passes, number 4 NT k + p: tokens 8 (p / 4) + p % 4 and the
            // fourth after it, a lane four rows of every fourth slice (the loads of eight lanes fall into different banks). A
            // fixed order of additions. The set's warps take turns with the passes.
            constexpr int kPasses = 4 * NT, kMine = (kMaxSlices + 3) / 4;
            const float *pass_src = parts + (lane >> 3) * kPart + (lane & 4) * kTokenPitch + (lane & 3) * 4;
            int pass = slice;
            auto add_passes = [&](int end) {
                for (; pass < end; pass += n_slices) {
                    const int k = pass / kPasses, p = pass % kPasses, token = 8 * (p >> 2) + (p & 3);
                    const float *src = pass_src + k % kBufs * (prm.slices * kPart) + token * kTokenPitch;
                    float4 total = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
                    for (int s = 0; s < kMine; ++s)
                        if (4 * s + (lane >> 3) < n_slices) total = add4(total, *reinterpret_cast<const float4 *>(src + 4 * s * kPart));
                    __syncwarp();
                    total = join4(total);
                    if (lane < 8) {
                        const int i = subset + k * prm.subsets, m = token + (lane & 4), row = (lane & 3) * 4;
                        if (split_log == 0) {
                            store_rows(prm, (tile_lo + i) * kTileRows + row, m, total);
                        } else {                                // to CTA i % split of the cluster, which adds the CTAs' sums
                            const int slot = (i >> split_log << split_log) + rank;
                            uint32_t dst, bar;
                            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst)
                                         : "r"(base + prm.sums_addr + 4u * (uint32_t)(slot * kPart + m * kTokenPitch + row)), "r"(i & (split - 1)));
                            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(bar) : "r"(tile_bar(i >> split_log)), "r"(i & (split - 1)));
                            asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
                                         ::"r"(dst), "r"(__float_as_uint(total.x)), "r"(__float_as_uint(total.y)),
                                           "r"(__float_as_uint(total.z)), "r"(__float_as_uint(total.w)), "r"(bar) : "memory");
                        }
                    }
                    __syncwarp();
                }
            };
            auto run = [&](auto half_tag) {
                constexpr int HALF = decltype(half_tag)::value;
                int stage = subset, k = 0;
                uint32_t phase = 0;
                for (int i = subset; i < n_tiles; i += prm.subsets, ++k) {
                    uint32_t w_lo[7], w_hi[7];                  // this lane's words of both rows
                    mbar_wait(full_bar(stage), phase, prm.status, dead);
                    const uint32_t src = lane_src + (uint32_t)stage * stage_bytes;
                    auto words = [&](uint32_t (&w)[7], uint32_t at) {
                        w[0] = lds<0>(at);
                        if (HS == 2 || HALF == 0) { w[1] = lds<4>(at); w[2] = lds<8>(at); }
                        w[3] = lds<12>(at);
                        if (HS == 2 || HALF == 1) { w[4] = lds<16>(at); w[5] = lds<20>(at); w[6] = lds<24>(at); }
                    };
                    words(w_lo, src);
                    words(w_hi, src + row8);
                    __syncwarp();
                    if (lane == 0) mbar_arrive(empty_bar(stage));
                    stage += prm.subsets;
                    if (stage >= prm.stages) { stage -= prm.stages; phase ^= 1u; }
                    auto pool = [](uint32_t w) { return prmt(w, w ^ 0x8000u, 0x0510u); };       // [s_lo, s_hi, s_hi ^ 0x80]
                    float sum[NT][4];
                    {
                        const Decoder lo{w_lo, pool(w_lo[0]), even_entry, odd_entry}, hi{w_hi, pool(w_hi[0]), even_entry, odd_entry};
                        half_slice<NT, HALF, true>(lo, hi, b[0], sum);
                        if (HS == 2) half_slice<NT, 1, false>(lo, hi, b[HS - 1], sum);
                    }
                    // The set's tile kLag before this one is complete by now, or soon will be. That every warp has stored its
                    // sums of that tile also says that all passes of the one kLag before it are over, whose buffer this tile
                    // takes.
                    if (k >= kLag) {
                        mbar_wait(own_sum_bar + 8u * (uint32_t)((k - kLag) % kBufs), (uint32_t)((k - kLag) / kBufs) & 1u, prm.status, dead);
                        add_passes((k - kLag + 1) * kPasses);
                    }
                    float *dst = lane_dst + k % kBufs * (prm.slices * kPart);
#pragma unroll
                    for (int t = 0; t < NT; ++t) {
                        float *f = dst + t * kTokenTile;
                        f[0] = sum[t][0];
                        f[kTokenPitch] = sum[t][1];
                        f[8] = sum[t][2];
                        f[kTokenPitch + 8] = sum[t][3];
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(own_sum_bar + 8u * (uint32_t)(k % kBufs));
                }
                for (int j = k < kLag ? 0 : k - kLag; j < k; ++j) {
                    mbar_wait(own_sum_bar + 8u * (uint32_t)(j % kBufs), (uint32_t)(j / kBufs) & 1u, prm.status, dead);
                    add_passes((j + 1) * kPasses);
                }
            };
            if (HS == 1 && (half0 & 1)) run(std::integral_constant<int, 1>{});
            else run(std::integral_constant<int, 0>{});
        }
    }
    if (dead)                                                   // a wait ran out: give the copies still in flight time to land
        for (int i = 0; i < 64; ++i) __nanosleep(20000);
    if (split > 1) {
        // CTA r of the cluster has the CTAs' sums of every split-th tile; it adds them in the order of the columns as they come in
        // (with a cluster barrier before all of them 3 tokens of 264x17408 took 4.8 us, now 4.4; 8 of 640x8704 5.3 and 4.6; 12 of
        // 1024x5120 5.6 and 5.3)
        const float *sums = reinterpret_cast<const float *>(smem + (prm.sums_addr - kWindow));
        for (int j = warp; rank + (j / (4 * NT) << split_log) < n_tiles; j += warps) {
            const int own = j / (4 * NT), p = j % (4 * NT), m = 8 * (p >> 2) + (p & 3) + (lane & 4), row = (lane & 3) * 4;
            mbar_wait(tile_bar(own), 0, prm.status, dead);
            float4 total = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            for (int c = lane >> 3; c < split; c += 4)
                total = add4(total, *reinterpret_cast<const float4 *>(sums + ((own << split_log) + c) * kPart + m * kTokenPitch + row));
            __syncwarp();
            total = join4(total);
            if (lane < 8) store_rows(prm, (tile_lo + rank + (own << split_log)) * kTileRows + row, m, total);
        }
        if (dead) stay_with_cluster();
    }
}

// ---- host ---------------------------------------------------------------------------------------------------------
struct SlicePlan {
    bool ok;
    float us;
    int split, slices, subsets, clusters, stages, pitch;
    int x_bufs;
    uint32_t sums_addr, ring_addr, end;
};

KernelRecord g_records[2];                                      // of slices_kernel<1> and <2>
const void *kernel_of(int nt) {
    return nt == 1 ? reinterpret_cast<const void *>(slices_kernel<1>) : reinterpret_cast<const void *>(slices_kernel<2>);
}

// Modelled time (us) by which a K split is chosen: what the SM works through (0.128 per row tile and chunk of eight tokens, twice
// that for sixteen), or where there are few warps what one of them does one tile after the other, behind launch, table and
// activations; a cluster's barriers and its exchange on top.
float slice_us(int split, int slices, int per_cluster) {
    const int subsets = kMaxSlices / slices < per_cluster ? kMaxSlices / slices : per_cluster;
    const float sm = 0.128f * (float)(per_cluster * slices), chain = 0.7f * (float)((per_cluster + subsets - 1) / subsets);
    return (split > 1 ? 5.2f : 3.6f) + (sm > chain ? sm : chain);
}

// The K split with the smallest modelled time.
SlicePlan slice_plan(int nt, int N, int K, const int *rooms = nullptr) {
    SlicePlan best = {};
    const int per = slice_halves(nt), halves = K / 256 / per, tiles = (N + kTileRows - 1) / kTileRows;
    for (int log = 0; log <= 3; ++log) {
        const int split = 1 << log;
        SlicePlan p = {};
        p.split = split;
        p.slices = (halves + split - 1) / split;
        if (halves < split || p.slices > kMaxSlices) continue;
        // how many clusters run at once is asked of the driver (milliseconds, the first time) only where this split could win
        if (best.ok && slice_us(split, p.slices, (tiles + sm_count() / split - 1) / (sm_count() / split)) >= best.us) continue;
        const int room = rooms ? rooms[split] : clusters_at_once(g_records[nt - 1], kernel_of(nt), 32 * (kMaxSlices + kExtraWarps),
                                                                 kWindowEnd - kWindow, split);
        if (room < 1) continue;
        p.clusters = tiles < room ? tiles : room;
        const int per_cluster = (tiles + p.clusters - 1) / p.clusters;
        p.subsets = kMaxSlices / p.slices;
        if (p.subsets > per_cluster) p.subsets = per_cluster;
        // a CTA's slices may begin and end inside a chunk
        const int most = per == 2 ? p.slices : (p.slices + 2) / 2, chunks = most < K / 512 ? most : K / 512;
        p.pitch = chunks * kChunkBytes;
        if (p.pitch / 16 % 2 == 0) p.pitch += 16;
        p.x_bufs = p.subsets == 1 && nt == 2 ? 1 : 2;           // sets of warps share a slice's activations: all at once
        const auto aligned = [](int bytes) { return (uint32_t)(bytes + 127) / 128 * 128; };
        const uint32_t x_room = (uint32_t)(p.slices * p.x_bufs) * kXBytes;
        const uint32_t part_room = aligned(kBufs * p.subsets * p.slices * part_floats(nt) * 4);
        p.sums_addr = kDataAddr + (x_room > part_room ? x_room : part_room);
        p.ring_addr = p.sums_addr + (split > 1 ? aligned((per_cluster + split - 1) / split * split * part_floats(nt) * 4) : 0u);
        const uint32_t stage_bytes = (uint32_t)(kTileRows * p.pitch);
        p.stages = p.ring_addr < kWindowEnd ? (int)((kWindowEnd - p.ring_addr) / stage_bytes) : 0;
        if (p.stages > kMaxStages) p.stages = kMaxStages;
        if (p.stages > per_cluster) p.stages = per_cluster;
        if (p.stages < (per_cluster < 2 * p.subsets ? per_cluster : p.subsets + 1)) continue;      // no room to fetch ahead
        if (p.stages < per_cluster) {
            // A stage belongs to one set of warps: a wait for a barrier's parity tells a phase from the one before it only, so who
            // waits has to have seen that one.
            while (p.subsets > 1 && p.stages < 2 * p.subsets) --p.subsets;
            p.stages -= p.stages % p.subsets;
        }
        if (split > 1 && (per_cluster + split - 1) / split > kMaxOwn) continue;
        p.end = p.ring_addr + (uint32_t)p.stages * stage_bytes;
        p.ok = true;
        p.us = slice_us(split, p.slices, per_cluster);
        if (!best.ok || p.us < best.us) best = p;
    }
    return best;
}

// Modelled time (us) of a call behind another kernel, which this kernel has to beat the tcgen05 kernel at too: it gains 2 us from
// a call of this library before it, that one 1. Fitted to 1022 calls, weights out of HBM, within 6% (2-norm): launch, table and
// activations, a cluster's exchange, the turns of the sets of warps and the row tiles that go through a CTA. Of these calls the
// kernel that is chosen is within 2% of the better one, both in a row and apart, for all but 32, and never 9% behind in either
// (beyond eight tokens the line lies where it would lose as much to leave this kernel, 20% in a row, as to take it).
float call_us(const SlicePlan &p, int nt, int tiles) {
    const int per = (tiles + p.clusters - 1) / p.clusters, turns = (per + p.subsets - 1) / p.subsets;
    const float exchange = p.split == 1 ? 0.0f : p.split == 2 ? (nt == 1 ? 1.58f : 1.82f)
                         : p.split == 4 ? (nt == 1 ? 0.93f : 1.29f) : (nt == 1 ? 0.58f : 0.93f);
    return nt == 1 ? 4.47f + exchange + 0.329f * (float)turns + (float)per * (0.153f + 0.104f * (float)p.slices)
                   : 4.47f + exchange + 0.624f * (float)turns + (float)per * (0.231f + 0.043f * (float)p.slices);
}

template <int NT>
int launch_slices(const CUtensorMap &wmap, const CUtensorMap &xmap, const SliceParams &prm, const SlicePlan &p, cudaStream_t stream) {
    auto kern = slices_kernel<NT>;
    const cudaError_t e = opt_in(g_records[NT - 1], kernel_of(NT), kWindowEnd - kWindow);
    if (e != cudaSuccess) return cuda_fail(e, "tq1_linear_f16: shared memory opt-in (slices)");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(p.clusters * p.split));
    const int warps = prm.workers + kExtraWarps;
    cfg.blockDim = dim3((unsigned)(32 * (warps > kFillWarps ? warps : kFillWarps)));
    cfg.dynamicSmemBytes = p.end - kWindow;
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
    const cudaError_t err = cudaLaunchKernelEx(&cfg, kern, wmap, xmap, prm);
    if (captured && err == cudaSuccess) note_captured_kernel(stream);
    return err == cudaSuccess ? TQ1_OK : cuda_fail(err, "tq1_linear_f16: launch (slices)");
}

}  // namespace

// The plan of a call, not `ok` where the tcgen05 kernel is preferred.
static SlicePlan preferred_plan(int M, int N, int K) {
    if (M < 3 || M > 16 || K % 512 || gemm_tc_forced()) return {};
    const int nt = M <= 8 ? 1 : 2;
    SlicePlan p = slice_plan(nt, N, K);
    p.ok = p.ok && call_us(p, nt, (N + kTileRows - 1) / kTileRows) < (nt == 1 ? 1.0f : 1.04f) * gemm_tc_few_us(N, K);
    return p;
}

bool gemm_slices_layout(int M, int N, int K, const int *rooms, CallLayout *layout) {
    if (M < 3 || M > 16 || K % 512) return false;
    const SlicePlan p = slice_plan(M <= 8 ? 1 : 2, N, K, rooms);
    if (!p.ok) return false;
    *layout = {p.split, p.subsets, p.stages, ((N + kTileRows - 1) / kTileRows + p.clusters - 1) / p.clusters, gemm_slices_preferred(M, N, K)};
    return true;
}

bool gemm_slices_preferred(int M, int N, int K) { return preferred_plan(M, N, K).ok; }

static int launch_plan(const SlicePlan &p, const uint8_t *blocks, const __half *x, void *y, bool y_f32, int M, int N, int K,
                       void *workspace, cudaStream_t stream, bool swiglu) {
    const int nt = M <= 8 ? 1 : 2;
    SliceParams prm;
    prm.y = y;
    prm.status = static_cast<unsigned *>(workspace);
    prm.M = M;
    prm.N = N;
    prm.chunks = K / 512;
    prm.tiles = (N + kTileRows - 1) / kTileRows;
    prm.clusters = p.clusters;
    prm.split_log = p.split == 1 ? 0 : p.split == 2 ? 1 : p.split == 4 ? 2 : 3;
    prm.slices = p.slices;
    prm.subsets = p.subsets;
    prm.workers = p.slices * p.subsets;
    prm.stages = p.stages;
    prm.pitch = p.pitch;
    prm.x_bufs = p.x_bufs;
    prm.sums_addr = p.sums_addr;
    prm.ring_addr = p.ring_addr;
    prm.y_f32 = y_f32 ? 1 : 0;
    prm.swiglu = swiglu ? 1 : 0;
    prm.wide_y = N % 4 == 0 && (reinterpret_cast<uintptr_t>(y) & (y_f32 ? 15 : 7)) == 0 ? 1 : 0;
    // A row as 8-byte elements; a box is the 16 rows of a tile and a CTA's K range, at most 16 bytes more (another CTA's, or
    // filled in past the row's end), so that rows lie an odd number of 16-byte units apart.
    // Activations as [M][K / 128][2][64]: a box is one half of the four groups of a chunk for eight tokens.
    const EncodeTiledFn encode = encode_tiled_fn();
    if (!encode) return fail(TQ1_ERR_CUDA, "tq1_linear_f16: cuTensorMapEncodeTiled is unavailable");
    CUtensorMap wmap, xmap;
    const cuuint64_t row_bytes = (cuuint64_t)prm.chunks * kChunkBytes;
    const cuuint64_t w_dims[2] = {row_bytes / 8, (cuuint64_t)N}, w_strides[1] = {row_bytes};
    const cuuint32_t w_box[2] = {(cuuint32_t)p.pitch / 8, kTileRows}, ones[4] = {1, 1, 1, 1};
    CUresult res = encode(&wmap, CU_TENSOR_MAP_DATA_TYPE_INT64, 2, const_cast<uint8_t *>(blocks), w_dims, w_strides, w_box, ones,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (res != CUDA_SUCCESS) return fail(TQ1_ERR_CUDA, "tq1_linear_f16: weight tensor map failed (%d)", (int)res);
    const cuuint64_t x_dims[4] = {64, 2, (cuuint64_t)K / kGroup, (cuuint64_t)M};
    const cuuint64_t x_strides[3] = {128, 256, (cuuint64_t)K * sizeof(__half)};
    const cuuint32_t x_box[4] = {64, 1, 4, 8};
    res = encode(&xmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<__half *>(x), x_dims, x_strides, x_box, ones,
                 CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                 CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (res != CUDA_SUCCESS) return fail(TQ1_ERR_CUDA, "tq1_linear_f16: activation tensor map failed (%d)", (int)res);
    return nt == 1 ? launch_slices<1>(wmap, xmap, prm, p, stream) : launch_slices<2>(wmap, xmap, prm, p, stream);
}

int launch_gemm_slices(const uint8_t *blocks, const __half *x, void *y, bool y_f32, int M, int N, int K, void *workspace,
                       cudaStream_t stream, bool swiglu) {
    const SlicePlan p = slice_plan(M <= 8 ? 1 : 2, N, K);
    if (!p.ok) return fail(TQ1_ERR_INVALID, "tq1_linear_f16: %dx%dx%d does not fit the slice kernel", M, N, K);
    return launch_plan(p, blocks, x, y, y_f32, M, N, K, workspace, stream, swiglu);
}

bool try_gemm_slices(const uint8_t *blocks, const __half *x, void *y, bool y_f32, int M, int N, int K, void *workspace,
                     cudaStream_t stream, bool swiglu, int *status) {
    const SlicePlan p = preferred_plan(M, N, K);
    if (p.ok) *status = launch_plan(p, blocks, x, y, y_f32, M, N, K, workspace, stream, swiglu);
    return p.ok;
}

}  // namespace tq1
