// What the kernels of the exact batch-1 product share: units of 16 rows x 4 groups, their decode and products, and the digit
// planes of the activations. The arithmetic is described in tq1_gemv_chain.cu.
#pragma once
#include "tq1_common.cuh"

namespace tq1 {

namespace {

constexpr int kTileRows = 16;
constexpr int kChunkGroups = 4;
constexpr int kChunkCols = kChunkGroups * kGroup;             // 512
constexpr int kChunkBytes = kChunkGroups * kBlockBytes;       // 112
constexpr int kUnitBytes = kTileRows * kChunkBytes;           // 1792
constexpr int kRegsPerSub = 18;                                // A/B registers per lane per sub-unit

// Per activation group, written by the warp that prepared it: 121 * (sum of the fifth-trit activations),
// 2^(E-21) for the group's exponent E, and how many of its activations are Inf (kGroupNan: one is NaN).
constexpr int kGroupNan = 1 << 30;
struct alignas(16) GroupConst {
    int sum;
    float pow;
    int bad;
    int pad;
};

template <uint32_t SEL>
__device__ __forceinline__ uint32_t prmt_imm(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "n"(SEL));
    return d;
}
// Ring-buffer words. Not volatile: the address depends on the value returned by the barrier wait,
// which keeps the loads behind it while leaving the compiler free to interleave the two sub-units.
template <int OFF>
__device__ __forceinline__ uint32_t lds_off(uint32_t addr) {
    uint32_t v;
    asm("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(addr), "n"(OFF));
    return v;
}
template <bool SIGNED_A, bool ZERO_C>
__device__ __forceinline__ void mma_bytes(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                          uint32_t b0, uint32_t b1) {
    if (ZERO_C) {
        if (SIGNED_A)
            asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
                : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
                : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0), "r"(0), "r"(0), "r"(0));
        else
            asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
                : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
    } else {
        if (SIGNED_A)
            asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
        else
            asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    }
}

// One lane-stream (half a block: 14 code-byte slots in four words, wa holding slots 0,1 in its
// upper half) becomes 18 A registers: 14 table entries (weights of trits 0..3 of each slot) and
// the four raw words (the code bytes themselves, paired with the fifth trit's activation).
template <int TABLE>
__device__ __forceinline__ void decode_stream(uint32_t wa, uint32_t wb, uint32_t wc, uint32_t wd,
                                              uint32_t lane_base, uint32_t (&r)[kRegsPerSub]) {
    r[0] = lds_off<TABLE>(prmt_imm<0x7624>(wa, lane_base));
    r[1] = lds_off<TABLE>(prmt_imm<0x7634>(wa, lane_base));
    r[2] = lds_off<TABLE>(prmt_imm<0x7604>(wb, lane_base));
    r[3] = lds_off<TABLE>(prmt_imm<0x7614>(wb, lane_base));
    r[4] = lds_off<TABLE>(prmt_imm<0x7624>(wb, lane_base));
    r[5] = lds_off<TABLE>(prmt_imm<0x7634>(wb, lane_base));
    r[6] = lds_off<TABLE>(prmt_imm<0x7604>(wc, lane_base));
    r[7] = lds_off<TABLE>(prmt_imm<0x7614>(wc, lane_base));
    r[8] = lds_off<TABLE>(prmt_imm<0x7624>(wc, lane_base));
    r[9] = lds_off<TABLE>(prmt_imm<0x7634>(wc, lane_base));
    r[10] = lds_off<TABLE>(prmt_imm<0x7604>(wd, lane_base));
    r[11] = lds_off<TABLE>(prmt_imm<0x7614>(wd, lane_base));
    r[12] = lds_off<TABLE>(prmt_imm<0x7624>(wd, lane_base));
    r[13] = lds_off<TABLE>(prmt_imm<0x7634>(wd, lane_base));
    r[14] = wa;
    r[15] = wb;
    r[16] = wc;
    r[17] = wd;
}

// The digit planes of a chunk, as B fragments. Lane 4n + q holds the k-slots of column n; columns 0..3 are the digit planes of the
// two groups that the lanes q = 0, 1 decode, columns 4..7 of those of q = 2, 3, and the k-slots of the other pair are zero, so
// sixteen lanes have planes: number cls * 8 + 2 * plane + h for q = 2 cls + h. Each has its registers (both sub-units') side by side,
// which makes nine 16-byte loads of 36. 176 bytes from lane to lane: no bank conflicts there nor among the stores of a group.
constexpr int kPlaneLane = 176;
constexpr int kPlaneChunk = 16 * kPlaneLane;
static_assert(2 * kRegsPerSub * 4 <= kPlaneLane && kPlaneLane % 32 == 16, "planes of a lane");
// Where the planes of group gi of a chunk begin: sub-unit gi & 1, lanes q = 2 (gi >> 1) and the next.
__device__ __forceinline__ int plane_group(int gi) { return (gi & 1) * (kRegsPerSub * 4) + ((gi >> 1) & 1) * (8 * kPlaneLane); }
// B registers of both sub-units from the planes of a chunk at `planes` (shared window).
__device__ __forceinline__ void load_planes(uint32_t (&b)[2 * kRegsPerSub], uint32_t planes, int lane) {
    const int n = lane >> 2, cls = (lane >> 1) & 1;
    const bool live = (n >> 2) == cls;
    const uint32_t src = planes + (uint32_t)((cls * 8 + (n & 3) * 2 + (lane & 1)) * kPlaneLane);
#pragma unroll
    for (int i = 0; i < 2 * kRegsPerSub; i += 4) {
        b[i] = b[i + 1] = b[i + 2] = b[i + 3] = 0u;
        if (live)
            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(b[i]), "=r"(b[i + 1]), "=r"(b[i + 2]), "=r"(b[i + 3]) : "r"(src + 4u * i) : "memory");
    }
}

// One warp prepares G groups side by side, of which the first `live` are wanted. A group comes with four activations per lane
// (lane + 32 k, or with SIDE 4 lane + k): group maximum and fixed point. Then lane j < 26 takes the activations of code byte j
// (xchg: 128 words per group of the warp's own): the four that are paired with trits 0..3 make one register of each digit plane,
// whose place is the byte's slot in its half-block; the fifth is paired with the raw byte. (With a byte store per digit, sixteen
// a lane, a group took an SM 110 clocks.)
template <int G, bool SIDE>
__device__ __forceinline__ void prepare_groups(const float (&xv)[G][4], int live, int lane, int *xchg, unsigned char *const (&planes)[G],
                                               GroupConst *const (&results)[G]) {
    int e_biased[G], group_bad[G], e[G][5];
#pragma unroll
    for (int n = 0; n < G; ++n) {
        // non-negative floats order like their bit patterns: one redux instruction for the group maximum
        unsigned mbits = 0u;
        bool bad[4], anybad = false;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float a = fabsf(xv[n][k]);
            bad[k] = !(a <= 65504.0f);                         // NaN or Inf
            anybad = anybad || bad[k];
            mbits = max(mbits, bad[k] ? 0u : __float_as_uint(a));
        }
        mbits = __reduce_max_sync(0xffffffffu, mbits);
        // 2^E <= m < 2^(E+1); fixed point xi = round(v * 2^(21-E)), |xi| <= 2^22
        e_biased[n] = mbits != 0u ? (int)(mbits >> 23) : 127;
        const float up = __uint_as_float((uint32_t)(275 - e_biased[n]) << 23);             // 2^(21-E)
        int xi[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) xi[k] = __float2int_rn(xv[n][k] * up);
        group_bad[n] = __any_sync(0xffffffffu, anybad);        // infinite activations, or kGroupNan
        if (group_bad[n]) {                                    // rare; a finite group executes nothing of this
            int infs = 0;
            bool nan = false;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                infs += bad[k] ? 1 : 0;
                nan = nan || xv[n][k] != xv[n][k];
                xi[k] = bad[k] ? (xv[n][k] < 0.0f ? -1 : 1) : 0;
            }
            infs = __reduce_add_sync(0xffffffffu, infs);
            group_bad[n] = __any_sync(0xffffffffu, nan) ? kGroupNan : infs;
        }
        if (SIDE) {
            *reinterpret_cast<int4 *>(xchg + n * kGroup + 4 * lane) = make_int4(xi[0], xi[1], xi[2], xi[3]);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) xchg[n * kGroup + lane + 32 * k] = xi[k];
        }
    }
    __syncwarp();
    const int j = min(lane, 25), hh = j < 14 ? 0 : 1, slot = hh ? j - 12 : j;      // hh: which half-block lane decodes the byte
    const int place = hh * kPlaneLane + slot * 4;
    const int fifth_place = hh * kPlaneLane + (slot < 2 ? 14 * 4 + slot + 2 : 15 * 4 + slot - 2);
#pragma unroll
    for (int n = 0; n < G; ++n)
#pragma unroll
        for (int i = 0; i < 5; ++i) e[n][i] = i < 3 || j < 25 ? xchg[n * kGroup + 5 * j + i] : 0;      // the tail byte has three trits
#pragma unroll
    for (int n = 0; n < G; ++n) {
        // The values paired with the byte's trits, 81 x_i - 3^i x_4, and with the byte, x_4, as four signed byte digits: the bytes
        // of v + 0x80808080 are the digits plus 128.
        const int x4 = e[n][4];
        uint32_t v[5] = {(uint32_t)(81 * e[n][0] - x4), (uint32_t)(81 * e[n][1] - 3 * x4), (uint32_t)(81 * e[n][2] - 9 * x4),
                         (uint32_t)(81 * e[n][3] - 27 * x4), (uint32_t)x4};
#pragma unroll
        for (int i = 0; i < 5; ++i) v[i] = (v[i] + 0x80808080u) ^ 0x80808080u;
        const uint32_t a0 = prmt_imm<0x5140>(v[0], v[1]), a1 = prmt_imm<0x5140>(v[2], v[3]);
        const uint32_t a2 = prmt_imm<0x7362>(v[0], v[1]), a3 = prmt_imm<0x7362>(v[2], v[3]);
        const uint32_t plane[4] = {prmt_imm<0x5410>(a0, a1), prmt_imm<0x7632>(a0, a1), prmt_imm<0x5410>(a2, a3), prmt_imm<0x7632>(a2, a3)};
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            if (lane < 26 && n < live) *reinterpret_cast<uint32_t *>(planes[n] + place + p * 2 * kPlaneLane) = plane[p];
            if (lane < 25 && n < live) planes[n][fifth_place + p * 2 * kPlaneLane] = (unsigned char)(v[4] >> (8 * p));
        }
    }
#pragma unroll
    for (int n = 0; n < G; ++n) {
        const int s5 = __reduce_add_sync(0xffffffffu, lane < 25 ? 121 * e[n][4] : 0);              // 121 * sum of the fifth-trit activations
        if (lane == 0 && n < live) {
            GroupConst gc;
            gc.sum = s5;
            gc.pow = __uint_as_float((uint32_t)(e_biased[n] - 21) << 23);                          // 2^(E-21)
            gc.bad = group_bad[n];
            gc.pad = 0;
            *results[n] = gc;
        }
    }
}

}  // namespace

}  // namespace tq1
