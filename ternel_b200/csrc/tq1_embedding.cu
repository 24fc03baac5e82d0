// Packed-embedding row gather: out[t][k] = (c[id_t][k] - 1) * scale[id_t][k/128].
//
// Stands in for tq1_get_rows (src/ternel_mlx/kernels.py:863-901 of the reference)
// and k_get_rows_tq1_g128 (patches/prism-tq1-g128-distribution.patch:132-171).
// HBM-bound: per token it reads K/128*28 bytes and writes 2K (FP16) bytes.
//
// Sixteen threads decode one 28-byte block into 128 outputs, eight consecutive outputs (one 16-byte
// FP16 store, or two for FP32) per thread; a warp therefore writes 512 contiguous bytes. A thread's
// eight trits start somewhere inside a code byte and span at most three: the bytes are looked up in a
// table of five nibbles (twice the trit), joined and shifted, so that one multiply-add turns
// every second nibble into a byte-permute selector. Every output is one of three values per block, -1*s, 0*s, +1*s,
// computed once by multiplication (so that 0*Inf and 0*NaN give NaN and zeros keep the sign NumPy gives them) and
// then selected by the trit.
//
// What bounds it: up to a wave or two of CTAs the chain id -> code bytes -> table entries -> store, beyond that the stores
// (8192 tokens of 5120 columns: 21.4 us = 4.35 TB/s in FP16, 38.8 us = 4.56 TB/s in FP32). 2-bit trits unpacked one by one
// took 123 instructions per eight outputs: 6.5 us for 2048 tokens against 6.06 now, 23.1 for 8192.
#include "tq1_common.cuh"

namespace tq1 {

namespace {

struct TritTable {
    uint32_t e[256];
};
constexpr TritTable make_trit_table() {
    TritTable t{};
    for (int v = 0; v < 243; ++v) {
        int x = v;
        for (int i = 0; i < 5; ++i) {
            t.e[v] |= (uint32_t)(2 * (x % 3)) << (4 * i);
            x /= 3;
        }
    }
    return t;
}
__device__ const TritTable g_trits = make_trit_table();

constexpr int kThreadsPerBlockRow = 16;       // threads per 28-byte block
constexpr int kBlocksPerCta = 8;
constexpr int kTokensPerThread = 4;

}  // namespace

// SHARED: a CTA first copies the table to shared memory, which the few CTAs of a short call gain from; in a long one the
// barrier behind the copy costs more than lookups through L1 (launch_embedding has the line and the figures).
// DEPENDENT: the form for a programmatic dependent launch, of a short call: a long one gains nothing from that and loses from
// the plain loads (8192 tokens, FP32: 38.7 us, 42.7 with both). The ordinary form asks for the ids before the table, whose copy
// the dependent one has done by the time that the kernel before it ends.
template <bool OUT_F32, bool SHARED, bool DEPENDENT>
__global__ void __launch_bounds__(kThreadsPerBlockRow * kBlocksPerCta)
embedding_kernel(const uint8_t *blocks, const int64_t *ids, void *out,
                 int64_t T, int64_t V, int gpr) {
    const int j = threadIdx.x & (kThreadsPerBlockRow - 1);      // which eight outputs of the block
    const int g = blockIdx.x * kBlocksPerCta + (threadIdx.x >> 4);
    const bool in_row = g < gpr;                                // threads past the row only help to fill the table
    __shared__ uint32_t shared_trits[SHARED ? 256 : 1];
    const uint32_t *trits = SHARED ? shared_trits : g_trits.e;
    const int k0 = 8 * j;
    const int a = (k0 * 205) >> 10, off = k0 - 5 * a;            // k0 / 5 for k0 <= 120; first trit inside byte a
    const int64_t t0 = (int64_t)blockIdx.y * kTokensPerThread;

    // Several tokens per thread, every load of one kind issued for all of them before the next kind:
    // the dependent chain id -> code bytes -> table entries is a few microseconds long, and a thread
    // that follows it for one token only keeps too few bytes in flight to fill the memory system.
    int64_t id[kTokensPerThread];
    bool live[kTokensPerThread];
    auto load_ids = [&] {
#pragma unroll
        for (int q = 0; q < kTokensPerThread; ++q)
            id[q] = in_row && t0 + q < T ? load_input<DEPENDENT>(reinterpret_cast<const long long *>(ids) + t0 + q) : -1;
    };
    if (!DEPENDENT) load_ids();
    if (SHARED) {
#pragma unroll
        for (int i = 0; i < 256; i += kThreadsPerBlockRow * kBlocksPerCta)
            shared_trits[i + threadIdx.x] = g_trits.e[i + threadIdx.x];
    }
    if (DEPENDENT) {
        grid_dependency_wait();
        load_ids();
    }
    const uint8_t *blk[kTokensPerThread];
    uint32_t sbits[kTokensPerThread], b0[kTokensPerThread], b1[kTokensPerThread], b2[kTokensPerThread];
#pragma unroll
    for (int q = 0; q < kTokensPerThread; ++q) {
        live[q] = id[q] >= 0 && id[q] < V;
        blk[q] = blocks + (size_t)((unsigned)(live[q] ? id[q] : 0) * (unsigned)gpr + (unsigned)(in_row ? g : 0)) * kBlockBytes;
        sbits[q] = load_input<DEPENDENT>(reinterpret_cast<const unsigned short *>(blk[q]));
        b0[q] = load_input<DEPENDENT>(blk[q] + 2 + a);
        b1[q] = load_input<DEPENDENT>(blk[q] + 3 + a);
        b2[q] = off >= 3 ? load_input<DEPENDENT>(blk[q] + 4 + a) : 0u;  // the third byte exists whenever it is needed
    }
    if (SHARED) {
        __syncthreads();
        // not before the loads: CTAs of the next gather that wait beside this one's take places unevenly
        allow_next_grid();
    }
    if (!in_row) return;
    uint32_t sel[kTokensPerThread];                             // eight nibbles, output i at bits 4i..4i+3
#pragma unroll
    for (int q = 0; q < kTokensPerThread; ++q) {
        const uint32_t n0 = trits[b0[q]], n1 = trits[b1[q]], n2 = trits[b2[q]];
        sel[q] = __funnelshift_r(n0 | (n1 << 20), (n1 >> 12) | (n2 << 8), 4 * off);
    }
#pragma unroll
    for (int q = 0; q < kTokensPerThread; ++q) {
        if (t0 + q >= T) break;
        const __half scale = __ushort_as_half((unsigned short)sbits[q]);
        const size_t base = ((size_t)(t0 + q) * gpr + g) * kGroup + 8 * j;
        if (!TQ1_IN_BOUNDS(base + 7, (size_t)T * gpr * kGroup, 30u)) continue;
        if (OUT_F32) {
            // a row outside the table is all zeros, not 0 * scale
            const float sf = __half2float(scale);
            const float c0 = live[q] ? -1.0f * sf : 0.0f, c1 = live[q] ? 0.0f * sf : 0.0f, c2 = live[q] ? 1.0f * sf : 0.0f;
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint32_t trit2 = sel[q] >> (4 * i) & 15u;
                v[i] = trit2 == 0 ? c0 : trit2 == 2 ? c1 : c2;
            }
            float4 *dst = reinterpret_cast<float4 *>(static_cast<float *>(out) + base);
            dst[0] = make_float4(v[0], v[1], v[2], v[3]);
            dst[1] = make_float4(v[4], v[5], v[6], v[7]);
        } else {
            // The three candidate halves sit in an 8-byte pool. A trit t selects pool bytes 2t and 2t+1, selector nibbles
            // (2t, 2t+1): a nibble n in a byte of its own becomes 0x11 * n + 0x10.
            const __half2 c01 = __hmul2(__half2half2(scale), __floats2half2_rn(-1.0f, 0.0f));
            // 1 * s, which the compiler takes for s itself: a NaN scale gives the NaN 0x7fff that a multiplication gives
            const uint32_t c2 = __hisnan(scale) ? 0x7fffu : sbits[q];
            // a row outside the table is all zeros, not 0 * scale
            const uint32_t pool_lo = live[q] ? reinterpret_cast<const uint32_t &>(c01) : 0u;
            const uint32_t pool_hi = live[q] ? c2 : 0u;
            const uint32_t even = (sel[q] & 0x0f0f0f0fu) * 0x11u + 0x10101010u;
            const uint32_t odd = (sel[q] >> 4 & 0x0f0f0f0fu) * 0x11u + 0x10101010u;
            uint32_t w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
                w[i] = __byte_perm(pool_lo, pool_hi, __byte_perm(even, odd, 0x40u + 0x11u * i));
            *reinterpret_cast<uint4 *>(static_cast<__half *>(out) + base) = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
}

// Up to this many CTAs (two waves of sixteen per SM) the table goes through shared memory: 512 / 2048 / 8192 tokens of 5120
// columns, FP16, take 3.03 / 6.06 / 22.7 us with it and 3.21 / 6.12 / 21.4 without; FP32 5.06 / 12.9 / 43.3 and
// 5.23 / 13.7 / 38.8.
constexpr long long kSharedTableCtas = 2 * 16 * 148;

int launch_embedding(const uint8_t *blocks, const int64_t *ids, void *out, bool out_f32,
                     int64_t T, int64_t V, int K, cudaStream_t stream) {
    const int gpr = K / kGroup;
    const int64_t per_launch = 65535LL * kTokensPerThread;          // gridDim.y limit
    for (int64_t t0 = 0; t0 < T; t0 += per_launch) {
        const int64_t n = T - t0 < per_launch ? T - t0 : per_launch;
        dim3 grid((gpr + kBlocksPerCta - 1) / kBlocksPerCta, (unsigned)((n + kTokensPerThread - 1) / kTokensPerThread));
        const bool shared = (long long)grid.x * grid.y <= kSharedTableCtas;
        void *first = out_f32 ? static_cast<void *>(static_cast<float *>(out) + t0 * K)
                              : static_cast<void *>(static_cast<__half *>(out) + t0 * K);
        auto dependent = out_f32 ? embedding_kernel<true, true, true> : embedding_kernel<false, true, true>;
        auto plain = out_f32 ? (shared ? embedding_kernel<true, true, false> : embedding_kernel<true, false, false>)
                             : (shared ? embedding_kernel<false, true, false> : embedding_kernel<false, false, false>);
        const cudaError_t err = launch_either(shared, shared, shared, dependent, plain, grid, kThreadsPerBlockRow * kBlocksPerCta, 0, stream, blocks,
                                              ids + t0, first, n, V, gpr);
        if (err != cudaSuccess) return cuda_fail(err, "tq1_embedding_f16: launch");
    }
    return TQ1_OK;
}

}  // namespace tq1
