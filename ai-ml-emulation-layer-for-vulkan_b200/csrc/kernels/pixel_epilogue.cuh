// The main RESCALE stage of the pixel-major tensor-core kernels (a thread holds 16 output columns of one pixel): the table of
// per-column constants in shared memory and the forms in which it is evaluated.
#ifndef MLEL_PIXEL_EPILOGUE_CUH
#define MLEL_PIXEL_EPILOGUE_CUH

#include <cstdint>

#include "device_common.cuh"

namespace mlel {
namespace tc {

// Constants of the main RESCALE stage for one output column (see FastRescale): two shared-memory reads per
// element, by shared address.  A table is built in one of two forms.  General: {mult, corr0, rnLo, rnHi} with the
// rounding constant for v < zpIn (input zero point folded in).  High-word form, when every shift of the table is
// at least 32 and the corrections are small (see scaleHigh): {mult, corr0 - zpIn, rnM} with the rounding constant
// without the zero-point fold.  32-bit form, when in addition every shift is at most 60 and the host has bounded
// |x| below 2^29 (see scaleHigh32): {mult, 4 * (corr0 - zpIn), rounding units, shift - 30} -- one read per element.
struct __align__(16) ColConst {
    int32_t mult;
    int32_t corr;        // general: correction of the most common border class; high-word form: that minus zpIn
    uint32_t rnLo, rnHi; // rounding constant (see above)
    int32_t s2;          // max(shift - 32, 0)
    uint32_t bump;       // what the constant for v >= zpIn adds: 2^31 with double rounding and shift > 31, else 0
    int32_t s1;          // min(shift, 32)
    int32_t corr0;       // correction of the most common border class (what a border pixel swaps for its own)
};

// High word of (accumulator + correction - zpIn) * mult + rounding: with x = v - zpIn the double-rounding test
// v >= zpIn is the sign of x, and bumpMask (2^31 or 0) & ~x adds the 2^31 for x >= 0.  The caller shifts the high
// word by shift - 32.  Exact while x does not overflow, which the host's bound on the corrections guarantees.
__device__ __forceinline__ int32_t scaleHigh(int32_t x, int32_t mult, uint64_t rn, uint32_t bumpMask) {
    const uint64_t prod = uint64_t(int64_t(x) * int64_t(mult));
    const uint32_t extra = ~uint32_t(x) & bumpMask;
    const uint64_t sum = prod + rn + uint64_t(extra);
    return int32_t(uint32_t(sum >> 32));
}

__device__ __forceinline__ void ldsV2(uint32_t addr, uint32_t &a, uint32_t &b) {
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(a), "=r"(b) : "r"(addr));
}
__device__ __forceinline__ int32_t ldsS32(uint32_t addr) {
    int32_t v;
    asm volatile("ld.shared.s32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void ldsV4(uint32_t addr, uint32_t &a, uint32_t &b, uint32_t &c, uint32_t &d) {
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(a), "=r"(b), "=r"(c), "=r"(d) : "r"(addr));
}

// Packs the low bytes of four int32 values, e0 in the lowest byte (values are already clamped to int8).
__device__ __forceinline__ uint32_t pack4(int32_t e0, int32_t e1, int32_t e2, int32_t e3) {
    const uint32_t lo = __byte_perm(uint32_t(e0), uint32_t(e1), 0x0040);
    const uint32_t hi = __byte_perm(uint32_t(e2), uint32_t(e3), 0x0040);
    return __byte_perm(lo, hi, 0x5410);
}

// 16 columns of one row in the 32-bit form of the constants table (see ColConst), packed four results to a word.
template <bool SIGNED>
__device__ __forceinline__ void rescale16Words32(const uint32_t (&acc)[16], uint32_t tabAddr, int32_t outZp, int32_t lo,
                                                 int32_t hi, uint32_t (&packed)[4]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        int32_t y[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int j = 4 * q + e;
            uint32_t mult, corrX4, c32, shift32;
            ldsV4(tabAddr + uint32_t(j) * 32u, mult, corrX4, c32, shift32);
            const int32_t x4 = int32_t(acc[j] * 4u + corrX4);
            const int32_t h = scaleHigh32<SIGNED>(x4, int32_t(mult), int32_t(c32));
            y[e] = min(__viaddmax_s32(h >> shift32, outZp, lo), hi);
        }
        packed[q] = pack4(y[0], y[1], y[2], y[3]);
    }
}

// The same in the general form.
__device__ __forceinline__ void rescale16General(const uint32_t (&acc)[16], uint32_t tabAddr, int32_t zpIn, int32_t outZp, int32_t lo,
                                                 int32_t hi, uint32_t (&packed)[4]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        int32_t y[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int j = 4 * q + e;
            uint32_t mult, corr, rnLo, rnHi, s2, bump;
            ldsV4(tabAddr + uint32_t(j) * 32u, mult, corr, rnLo, rnHi);
            ldsV2(tabAddr + uint32_t(j) * 32u + 16u, s2, bump);
            const uint32_t s1 = uint32_t(ldsS32(tabAddr + uint32_t(j) * 32u + 24u));
            const int32_t v = int32_t(acc[j] + corr);
            const uint64_t sum = uint64_t(int64_t(v) * int64_t(int32_t(mult))) + ((uint64_t(rnHi) << 32) | rnLo) +
                                 uint64_t(v >= zpIn ? bump : 0u);
            const int32_t q32 = int32_t(__funnelshift_rc(uint32_t(sum), uint32_t(sum >> 32), s1));
            y[e] = min(__viaddmax_s32(q32 >> s2, outZp, lo), hi);
        }
        packed[q] = pack4(y[0], y[1], y[2], y[3]);
    }
}

} // namespace tc
} // namespace mlel

#endif
