// Linear of two and more activation rows for the weights that the tcgen05 kernel does not take: widths that are no multiple
// of 512 and blocks that do not start on a 16-byte boundary.
//
// The arithmetic is the reference's: a full FP32 sum per 128-weight group, then acc = fma(scale, group_sum, acc)
// (src/bonsai_tq1/reference.py:33-38, src/ternel_mlx/kernels.py:317-322), so non-finite scales and activations come out as
// they do there. Weights stay -1, 0, +1 and enter mma.sync.m16n8k16 as its A operand; an accumulator covers 32 columns, the
// sums of those are FP32 additions on the CUDA cores. The tcgen05 kernel with 4-byte copies had taken these widths with one
// truncating accumulator over a whole K part: 1.3e-6 from the FP64 product (2-norm, 4099x2176) and 5.3e-6 (300 tokens of
// 17408x5248) where the row kernel is at 5.7e-8 and 7.2e-8; this one is at 4.2e-8 and 5.3e-8.
//
// The contraction may take the columns of a group in any order as long as both operands agree. Here lane q of a quad holds
// columns 32 s + 8 q .. + 7 of a group for two K = 16 steps: as activations that is one 16-byte load, as weights it is one
// decoding task of eight consecutive trits (at most three code bytes), whose four registers are the A fragments themselves.
// Decoded weights never pass through shared memory.
//
//   few    a CTA has 16 weight rows and 8 NT tokens; its eight warps take every eighth group, so that the whole chain of a
//          short call is load, decode, product and one sum through shared memory
//   many   a CTA has 128 weight rows and 8 NT tokens; activations come through shared memory (three stages of cp.async)
//
// What bounds it: the chain of dependent loads and the decode (25 instructions and six table or byte loads per eight weights).
// 5 tokens of 4099x2176 take 5.2 us in a row of calls (6.3 behind another kernel, 5.9 through the Python module; row kernel 45).
// A `many` CTA of 64 tokens is bound by its products (the mma.sync pipe is active for 57% of the time); most calls of that length
// go to the tcgen05 form (tq1_gemm_groups_tc.cu).
#include "tq1_common.cuh"

namespace tq1 {

namespace {

constexpr int kGroupRowWords = kBlockWords;     // packed words of one row and group

// Five trits of a byte as nibbles, twice the trit each (the embedding kernel's form).
struct GroupTable {
    uint32_t e[256];
};
constexpr GroupTable make_group_table() {
    GroupTable t{};
    for (int v = 0; v < 243; ++v) {
        int x = v;
        for (int i = 0; i < 5; ++i) {
            t.e[v] |= (uint32_t)(2 * (x % 3)) << (4 * i);
            x /= 3;
        }
    }
    return t;
}
__device__ const GroupTable g_group_table = make_group_table();

// Eight trits starting at trit `off` of byte `code[0]` as FP16 weights -1, 0, +1, two to a register.
__device__ __forceinline__ void decode8(const uint8_t *code, int off, const uint32_t *table, uint32_t (&w)[4]) {
    const uint32_t n0 = table[code[0]], n1 = table[code[1]], n2 = off >= 3 ? table[code[2]] : 0u;
    const uint32_t sel = __funnelshift_r(n0 | (n1 << 20), (n1 >> 12) | (n2 << 8), 4 * off);
    const uint32_t even = (sel & 0x0f0f0f0fu) * 0x11u + 0x10101010u;
    const uint32_t odd = (sel >> 4 & 0x0f0f0f0fu) * 0x11u + 0x10101010u;
#pragma unroll
    for (int i = 0; i < 4; ++i)
        w[i] = __byte_perm(0x0000bc00u, 0x00003c00u, __byte_perm(even, odd, 0x40u + 0x11u * i));
}

__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// One 32-column step of a row tile (rows lo and hi of this lane decoded) against eight tokens: added to the group's sums.
__device__ __forceinline__ void step32(float (&sum)[4], const uint32_t (&lo)[4], const uint32_t (&hi)[4], const uint4 &x) {
    const uint32_t a[4] = {lo[0], hi[0], lo[1], hi[1]}, b[4] = {lo[2], hi[2], lo[3], hi[3]};
    float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    mma16816(d, a, x.x, x.y);
    mma16816(d, b, x.z, x.w);
#pragma unroll
    for (int i = 0; i < 4; ++i) sum[i] += d[i];
}

__device__ __forceinline__ void store_result(void *y, int y_f32, size_t o, size_t limit, float v) {
    if (!TQ1_IN_BOUNDS(o, limit, 70u)) return;
    if (y_f32) static_cast<float *>(y)[o] = v;
    else static_cast<__half *>(y)[o] = __float2half_rn(v);
}

// NT: token tiles of eight per CTA; DEPENDENT: the form for a programmatic dependent launch.
constexpr int kFewWarps = 8, kFewRows = 16;

template <int NT, bool DEPENDENT>
__global__ void __launch_bounds__(kFewWarps * 32)
groups_few_kernel(const uint8_t *blocks, const __half *x, void *y, int y_f32,
                  int M, int N, int groups) {
    __shared__ uint32_t table[256];
    __shared__ uint32_t packed[kFewWarps][kFewRows * kGroupRowWords];
    __shared__ float parts[kFewWarps][8 * NT][kFewRows];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
    const int tiles_m = (M + 8 * NT - 1) / (8 * NT), tile_n = blockIdx.x / tiles_m;
    const int n0 = tile_n * kFewRows, m0 = (blockIdx.x - tile_n * tiles_m) * 8 * NT;
    table[tid] = g_group_table.e[tid];
    // this lane's words of a group: word i of the tile's 16 x 7 (rows past the end read the last row, unused)
    constexpr int kWords = kFewRows * kGroupRowWords, kPerLane = (kWords + 31) / 32;
    const uint32_t *src[kPerLane];
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) {
        const int i = min(lane + 32 * j, kWords - 1), row = min(n0 + i / kGroupRowWords, N - 1);
        src[j] = reinterpret_cast<const uint32_t *>(blocks + (size_t)row * groups * kBlockBytes) + i % kGroupRowWords;
    }
    const __half *xrow[NT];
    bool live[NT];
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        const int m = m0 + 8 * t + g;
        live[t] = m < M;
        xrow[t] = x + (size_t)(live[t] ? m : 0) * groups * kGroup + 8 * q;
    }
    float acc[NT][4];
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[t][i] = 0.0f;
    uint32_t next[kPerLane];
    auto load = [&](int grp) {
#pragma unroll
        for (int j = 0; j < kPerLane; ++j)
            next[j] = grp < groups ? load_input<DEPENDENT>(src[j] + (size_t)grp * kGroupRowWords) : 0u;
    };
    if (DEPENDENT) grid_dependency_wait();
    load(warp);
    __syncthreads();
    uint32_t *mine = packed[warp];
    const uint8_t *bytes_lo = reinterpret_cast<const uint8_t *>(mine + g * kGroupRowWords);
    const uint8_t *bytes_hi = reinterpret_cast<const uint8_t *>(mine + (g + 8) * kGroupRowWords);
    for (int grp = warp; grp < groups; grp += kFewWarps) {
#pragma unroll
        for (int j = 0; j < kPerLane; ++j)
            if (lane + 32 * j < kWords) mine[lane + 32 * j] = next[j];
        __syncwarp();
        load(grp + kFewWarps);
        float sum[NT][4], half[NT][4];                  // the group's sum so far, that of its second half
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int i = 0; i < 4; ++i) sum[t][i] = half[t][i] = 0.0f;
        uint4 xv[4][NT];
#pragma unroll
        for (int s = 0; s < 4; ++s)
#pragma unroll
            for (int t = 0; t < NT; ++t)
                xv[s][t] = live[t] ? load_input<DEPENDENT>(reinterpret_cast<const uint4 *>(xrow[t] + (size_t)grp * kGroup + 32 * s))
                                   : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const int trit = 32 * s + 8 * q, a = (trit * 205) >> 10, off = trit - 5 * a;       // trit / 5 for trit <= 120
            uint32_t lo[4], hi[4];
            decode8(bytes_lo + 2 + a, off, table, lo);
            decode8(bytes_hi + 2 + a, off, table, hi);
#pragma unroll
            for (int t = 0; t < NT; ++t) step32(s < 2 ? sum[t] : half[t], lo, hi, xv[s][t]);
        }
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int i = 0; i < 4; ++i) sum[t][i] += half[t][i];
        const float s_lo = __half2float(*reinterpret_cast<const __half *>(bytes_lo));
        const float s_hi = __half2float(*reinterpret_cast<const __half *>(bytes_hi));
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            acc[t][0] = fmaf(s_lo, sum[t][0], acc[t][0]);
            acc[t][1] = fmaf(s_lo, sum[t][1], acc[t][1]);
            acc[t][2] = fmaf(s_hi, sum[t][2], acc[t][2]);
            acc[t][3] = fmaf(s_hi, sum[t][3], acc[t][3]);
        }
        __syncwarp();                                   // the packed bytes have been read
    }
    // Not earlier: CTAs of the next call that wait beside this one's take places unevenly (8 tokens of 4099x2176 replayed in a
    // graph: 6.0 us without the dependent launch, 8.0 with an early one, 5.3 with this).
    allow_next_grid();
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        parts[warp][8 * t + 2 * q][g] = acc[t][0];
        parts[warp][8 * t + 2 * q + 1][g] = acc[t][1];
        parts[warp][8 * t + 2 * q][g + 8] = acc[t][2];
        parts[warp][8 * t + 2 * q + 1][g + 8] = acc[t][3];
    }
    __syncthreads();
    for (int i = tid; i < 8 * NT * kFewRows; i += kFewWarps * 32) {
        const int r = i % kFewRows, t = i / kFewRows;
        double v = 0.0;                                 // one rounding for the sum of the warps' parts
#pragma unroll
        for (int w = 0; w < kFewWarps; ++w) v += (double)parts[w][t][r];
        if (n0 + r < N && m0 + t < M)
            store_result(y, y_f32, (size_t)(m0 + t) * N + n0 + r, (size_t)M * N, (float)v);
    }
}

constexpr int kManyWarps = 8, kManyRows = 16 * kManyWarps, kManyStages = 3;
constexpr size_t many_smem(int nt) {
    return (size_t)kManyStages * 8 * nt * kGroup * 2 + kManyWarps * 16 * kBlockBytes + 1024;
}

template <int NT, bool DEPENDENT>
__global__ void __launch_bounds__(kManyWarps * 32, NT == 8 ? 1 : 2)
groups_many_kernel(const uint8_t *blocks, const __half *x, void *y, int y_f32,
                   int M, int N, int groups) {
    constexpr int kTokens = 8 * NT, kStageBytes = kTokens * kGroup * 2, kThreads = kManyWarps * 32;
    extern __shared__ __align__(128) unsigned char smem[];
    uint32_t *table = reinterpret_cast<uint32_t *>(smem + kManyStages * kStageBytes);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
    uint32_t *mine = table + 256 + warp * 16 * kGroupRowWords;
    const int tiles_m = (M + kTokens - 1) / kTokens, tile_n = blockIdx.x / tiles_m;
    const int n0 = tile_n * kManyRows + warp * 16, m0 = (blockIdx.x - tile_n * tiles_m) * kTokens;
    table[tid] = g_group_table.e[tid];

    const uint32_t stage0 = (uint32_t)__cvta_generic_to_shared(smem);
    // 16-byte piece c of token t lies at piece c ^ 4 (t & 1) of its row: the eight lanes of a phase of a 16-byte load have
    // two tokens and four neighbouring pieces
    auto request = [&](int grp) {
        const uint32_t stage = stage0 + (uint32_t)(grp % kManyStages) * kStageBytes;
#pragma unroll
        for (int j = 0; j < (kTokens * 16 + kThreads - 1) / kThreads; ++j) {
            const int i = tid + j * kThreads, t = i >> 4, c = i & 15;
            if (kTokens * 16 % kThreads && i >= kTokens * 16) break;
            const bool in = m0 + t < M && grp < groups;
            const __half *src = x + ((size_t)(in ? m0 + t : 0) * groups + (in ? grp : 0)) * kGroup + 8 * c;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                         ::"r"(stage + (uint32_t)(t * 256 + ((c ^ (4 * (t & 1))) << 4))), "l"(src), "r"(in ? 16 : 0) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    constexpr int kWords = 16 * kGroupRowWords, kPerLane = (kWords + 31) / 32;
    const uint32_t *src[kPerLane];                      // word lane + 32 j of the warp's 16 x 7
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) {
        const int i = min(lane + 32 * j, kWords - 1), row = min(n0 + i / kGroupRowWords, N - 1);
        src[j] = reinterpret_cast<const uint32_t *>(blocks + (size_t)row * groups * kBlockBytes) + i % kGroupRowWords;
    }
    uint32_t next[kPerLane];
    auto load = [&](int grp) {
#pragma unroll
        for (int j = 0; j < kPerLane; ++j)
            next[j] = grp < groups ? load_input<DEPENDENT>(src[j] + (size_t)grp * kGroupRowWords) : 0u;
    };
    if (DEPENDENT) grid_dependency_wait();
    load(0);
    request(0);
    request(1);
    // Four groups at a time are summed apart and added with the rounding error carried along (Kahan's summation): one
    // plain chain over all 41 groups of 5248 columns rounds to 1.2e-7, the row kernel's four chains to 7.2e-8.
    float acc[NT][4], carry[NT][4], part[NT][4];
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[t][i] = carry[t][i] = part[t][i] = 0.0f;

    const uint8_t *bytes_lo = reinterpret_cast<const uint8_t *>(mine + g * kGroupRowWords);
    const uint8_t *bytes_hi = reinterpret_cast<const uint8_t *>(mine + (g + 8) * kGroupRowWords);
    for (int grp = 0; grp < groups; ++grp) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                                // this group's activations are there; the stage before is free
        request(grp + 2);
#pragma unroll
        for (int j = 0; j < kPerLane; ++j)
            if (lane + 32 * j < kWords) mine[lane + 32 * j] = next[j];
        __syncwarp();
        load(grp + 1);
        const unsigned char *stage = smem + (size_t)(grp % kManyStages) * kStageBytes;
        float sum[NT][4];
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int i = 0; i < 4; ++i) sum[t][i] = 0.0f;
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const int trit = 32 * s + 8 * q, a = (trit * 205) >> 10, off = trit - 5 * a;
            uint32_t lo[4], hi[4];
            decode8(bytes_lo + 2 + a, off, table, lo);
            decode8(bytes_hi + 2 + a, off, table, hi);
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                const uint4 xv = *reinterpret_cast<const uint4 *>(stage + (8 * t + g) * 256 +
                                                                  (((4 * s + q) ^ (4 * (g & 1))) << 4));
                step32(sum[t], lo, hi, xv);
            }
        }
        const float s_lo = __half2float(*reinterpret_cast<const __half *>(bytes_lo));
        const float s_hi = __half2float(*reinterpret_cast<const __half *>(bytes_hi));
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int i = 0; i < 4; ++i) part[t][i] = fmaf(i < 2 ? s_lo : s_hi, sum[t][i], part[t][i]);
        if ((grp & 3) == 3 || grp + 1 == groups) {
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float v = __fsub_rn(part[t][i], carry[t][i]), total = __fadd_rn(acc[t][i], v);
                    const float error = __fsub_rn(__fsub_rn(total, acc[t][i]), v);
                    carry[t][i] = fabsf(error) <= 3.4028235e38f ? error : 0.0f;         // an infinite sum stays what it is
                    acc[t][i] = total;
                    part[t][i] = 0.0f;
                }
        }
        __syncwarp();                                   // the packed bytes have been read
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    allow_next_grid();                                  // not earlier, as above: 16 tokens of 17408x5248 took 62 us instead of 38
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int n = n0 + g + (i >> 1) * 8, m = m0 + 8 * t + 2 * q + (i & 1);
            if (n < N && m < M) store_result(y, y_f32, (size_t)m * N + n, (size_t)M * N, acc[t][i]);
        }
}

template <int NT>
int launch_few(const uint8_t *blocks, const __half *x, void *y, int y_f32, int M, int N, int groups, cudaStream_t stream) {
    const long long ctas = (long long)((N + kFewRows - 1) / kFewRows) * ((M + 8 * NT - 1) / (8 * NT));
    // around one CTA an SM, a call whose first CTAs find places beside the last of the one before takes two places on some SMs
    // (120 CTAs: 8.7 us alone, 10.1 as a dependent launch; 24 of them 5.9 and 5.3, 257 of them 6.0 and 5.3)
    // (nor does it gain in a graph with two token tiles, three CTAs an SM: between one and a half and two of them on an SM a few
    // places are left to the next call, and between three and five the plain loads weigh more. 16 tokens, calls in a row, ordinary /
    // dependent: 275 CTAs of 1408 columns 5.35 / 5.81, of 9856 22.6 / 24.6, 625 of 2176 13.6 / 14.6, 175 of 640 3.46 / 2.78. Outside
    // a graph, where the launch itself costs 2 us: 275 of 1408 6.3 / 6.0, of 9856 24.5 / 25.8, 625 of 2176 15.8 / 14.6)
    const long long sms = sm_count();
    const bool uneven = NT == 2 && ((2 * ctas > 3 * sms && ctas <= 2 * sms) || (ctas > 3 * sms && ctas <= 5 * sms && groups > 8));
    const bool overlap = ctas <= sms / 2 || ctas > sms;
    const cudaError_t err = launch_either(overlap, overlap && !uneven, true, groups_few_kernel<NT, true>, groups_few_kernel<NT, false>,
                                          dim3((unsigned)ctas), kFewWarps * 32, 0, stream, blocks, x, y, y_f32, M, N, groups);
    return err == cudaSuccess ? TQ1_OK : cuda_fail(err, "tq1_linear_f16: launch");
}

template <int NT>
int launch_many(const uint8_t *blocks, const __half *x, void *y, int y_f32, int M, int N, int groups, cudaStream_t stream) {
    const long long ctas = (long long)((N + kManyRows - 1) / kManyRows) * ((M + 8 * NT - 1) / (8 * NT));
    static KernelRecord records[2];
    cudaError_t err = opt_in(records[0], reinterpret_cast<const void *>(groups_many_kernel<NT, true>), many_smem(NT));
    if (err == cudaSuccess) err = opt_in(records[1], reinterpret_cast<const void *>(groups_many_kernel<NT, false>), many_smem(NT));
    if (err != cudaSuccess) return cuda_fail(err, "tq1_linear_f16: shared memory opt-in");
    err = launch_either(true, true, true, groups_many_kernel<NT, true>, groups_many_kernel<NT, false>, dim3((unsigned)ctas), kManyWarps * 32,
                        many_smem(NT), stream, blocks, x, y, y_f32, M, N, groups);
    return err == cudaSuccess ? TQ1_OK : cuda_fail(err, "tq1_linear_f16: launch");
}

}  // namespace

bool gemm_groups_preferred(int M, int N, int K) { return M >= 2 && (long long)M * N * K >= (1 << 20); }

// Which of the three takes a call, by modelled times (us) with weights out of HBM. Up to 32 tokens fitted to 400 calls behind
// another kernel, within 8% (few), 3% (many) and 5% (tcgen05 form), the choice 1% above the best on average:
//   few    a warp works through every eighth group; what it takes grows with the CTAs on an SM
//   many   a CTA's groups one after the other; only where it fills most SMs, and its sums are the least exact of the three
//          (5.3e-8, few 4.2e-8, tcgen05 form 4.0e-8), so the tcgen05 form is preferred to it up to 10% behind
// 16 tokens of 17408x5248 41 us few, 37.5 many, 32 tcgen05 form; 16 of 8192x8320 40, 55 and 28; 32 of 5120x17280 68, 172 and 58;
// 16 of 4099x2176 7.5, 16 and 9.1; 16 of 34816x640 15.8, 10.7 and 13.
// Beyond 32 tokens: a few row takes 1.1 or (two CTAs an SM) 2.1 a group of eight, many 1.68 a group, the tcgen05 form 1.13.
// Without a status word the tcgen05 form, which waits on barriers with a limit, is left out: nobody would learn of a wait that
// ran out.
int gemm_groups_form(int M, int N, int K, bool status) {
    if (M <= 8) return TQ1_FORM_GROUPS_FEW;
    const int sms = sm_count();
    const auto rounds = [](long long ctas, int at_once) { return (float)((ctas + at_once - 1) / at_once); };
    const long long few_tiles = (N + kFewRows - 1) / kFewRows, row_tiles = (N + kManyRows - 1) / kManyRows;
    const float groups = (float)(K / kGroup), turns = (float)((K / kGroup + 7) / 8);
    bool many;
    float us, behind = 1.0f;
    if (M <= 32) {
        const float per_sm = (float)few_tiles / (float)sms;
        us = M <= 16 ? 1.62f + turns * (0.494f + 0.264f * rounds(few_tiles, sms) + 0.366f * per_sm + 0.497f * rounds(few_tiles, 3 * sms))
                     : 2.03f + turns * (0.073f + 0.633f * rounds(few_tiles, sms) + 0.263f * per_sm + 0.563f * rounds(few_tiles, 2 * sms));
        const float many_us = M <= 16 ? 2.14f + groups * (0.04f + 0.80f * rounds(row_tiles, sms))
                                      : 2.41f + groups * (0.35f + 0.92f * rounds(row_tiles, sms));
        many = row_tiles * 100 >= sms * (M <= 16 ? 86 : 70) && many_us < us;
        if (many) { us = many_us; behind = 1.1f; }
    } else {
        const long long token_tiles = (M + 63) / 64, few_ctas = few_tiles * ((M + 31) / 32);
        many = 2 * row_tiles * token_tiles >= sms;
        us = 3.0f + (many ? groups * 1.68f * rounds(row_tiles * token_tiles, sms)
                          : turns * (few_ctas <= sms ? 1.1f : 2.1f * rounds(few_ctas, 2 * sms)));
    }
    if (status && gemm_groups_tc_us(M, N, K) < behind * us) return TQ1_FORM_GROUPS_TCGEN05;
    return many ? TQ1_FORM_GROUPS_MANY : TQ1_FORM_GROUPS_FEW;
}

int launch_gemm_groups(int form, const uint8_t *blocks, const __half *x, void *y, bool y_f32, int M, int N, int K, unsigned *status,
                       cudaStream_t stream) {
    const int groups = K / kGroup, f32 = y_f32 ? 1 : 0;
    switch (form) {
        case TQ1_FORM_GROUPS_TCGEN05:
            return launch_gemm_groups_tc(blocks, x, y, y_f32, M, N, K, status, stream);
        case TQ1_FORM_GROUPS_MANY:
            return M <= 16   ? launch_many<2>(blocks, x, y, f32, M, N, groups, stream)
                   : M <= 32 ? launch_many<4>(blocks, x, y, f32, M, N, groups, stream)
                             : launch_many<8>(blocks, x, y, f32, M, N, groups, stream);
        default:
            return M <= 8    ? launch_few<1>(blocks, x, y, f32, M, N, groups, stream)
                   : M <= 16 ? launch_few<2>(blocks, x, y, f32, M, N, groups, stream)
                             : launch_few<4>(blocks, x, y, f32, M, N, groups, stream);
    }
}

}  // namespace tq1
