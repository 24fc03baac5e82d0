// What the kernels share that turn code bytes into FP16 weights by a table of PRMT selectors in shared memory.
#pragma once
#include "tq1_async.cuh"

namespace tq1 {

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Bounded, as in the other kernels: after the limit status 3 is set and the thread waits for nothing any more.
static __device__ __noinline__ bool mbar_wait_more(uint32_t bar, uint32_t parity, unsigned *status) {
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
    if (!ok) atomicExch(status, 3u);
    return !ok;
}
__device__ __forceinline__ void mbar_wait(uint32_t bar, uint32_t parity, unsigned *status, bool &dead) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    if (!ok && !dead) dead = mbar_wait_more(bar, parity, status);
}

// Table entry of code byte v: PRMT selectors that pick FP16 weights out of [s_lo, s_hi, s_hi ^ 0x80] and zeros, one byte a trit.
//   even byte (its first trit in the lower half of a register): word0 = (t0,t1) | t4 << 16, word1 = (t2,t3)
//   odd byte: word0 = (t1,t2) | t0 << 16, word1 = (t3,t4)
// The 13 values past 242 decode to zero weights: a byte that escaped the load-time scan reads inside the table.
struct CodeTable { uint2 e[512]; };                             // entry of byte v: e[2 v] even, e[2 v + 1] odd
constexpr CodeTable make_code_table() {
    CodeTable t{};
    for (int v = 0; v < 256; ++v) {
        uint32_t c[5] = {0x44u, 0x44u, 0x44u, 0x44u, 0x44u};
        int rest = v;
        for (int d = 0; d < 5 && v < 243; ++d) {
            c[d] = rest % 3 == 0 ? 0x20u : rest % 3 == 1 ? 0x44u : 0x10u;
            rest /= 3;
        }
        t.e[2 * v].x = c[0] | (c[1] << 8) | (c[4] << 16);
        t.e[2 * v].y = c[2] | (c[3] << 8);
        t.e[2 * v + 1].x = c[1] | (c[2] << 8) | (c[0] << 16);
        t.e[2 * v + 1].y = c[3] | (c[4] << 8);
    }
    return t;
}
static __device__ __align__(16) const CodeTable g_code_table = make_code_table();

// Fills the shared table: sixteen copies of every entry, two entries of both forms (512 bytes) per warp and step, several
// loads in flight.
constexpr uint32_t kCodeTableBytes = 65536;
__device__ __forceinline__ void fill_code_table(unsigned char *table, int warp, int warps, int lane) {
    constexpr int kSteps = 128, kFlight = 8;
    for (int j0 = warp; j0 < kSteps; j0 += kFlight * warps) {
        uint2 e[kFlight];
#pragma unroll
        for (int j = 0; j < kFlight; ++j)
            if (j0 + j * warps < kSteps) e[j] = __ldg(&g_code_table.e[4 * (j0 + j * warps) + (lane >> 3)]);
#pragma unroll
        for (int j = 0; j < kFlight; ++j)
            if (j0 + j * warps < kSteps)
                *reinterpret_cast<uint4 *>(table + (j0 + j * warps) * 512 + lane * 16) = make_uint4(e[j].x, e[j].y, e[j].x, e[j].y);
    }
}

// A lane's 64 weights of one row, 32 registers of two, in the order of the columns. Eager: everything the caller's loop
// unrolls into; `w` holds the block's words (of half 0 words 0..3, of half 1 words 0 and 3..6).
template <uint32_t TABLE>
struct RowDecoder {
    const uint32_t *w;
    uint32_t pool, even_entry, odd_entry;
    __device__ __forceinline__ void lookup(int j, uint32_t &e0, uint32_t &e1) const {        // code byte j
        const uint32_t addr = prmt(w[(2 + j) >> 2], j & 1 ? odd_entry : even_entry, 0x7604u | (uint32_t)(((2 + j) & 3) << 4));
        asm("ld.shared.v2.u32 {%0, %1}, [%2+%3];" : "=r"(e0), "=r"(e1) : "r"(addr), "n"(TABLE));
    }
    __device__ __forceinline__ uint32_t pick(uint32_t sel) const { return prmt(pool, 0u, sel); }
    // ten weights of code bytes j (even) and j + 1
    __device__ __forceinline__ void two_bytes(int j, uint32_t *v) const {
        uint32_t e0, e1, f0, f1;
        lookup(j, e0, e1);
        lookup(j + 1, f0, f1);
        v[0] = pick(e0);
        v[1] = pick(e1);
        v[2] = pick(prmt(e0, f0, 0x0062));
        v[3] = pick(f0);
        v[4] = pick(f1);
    }
};

}  // namespace tq1
