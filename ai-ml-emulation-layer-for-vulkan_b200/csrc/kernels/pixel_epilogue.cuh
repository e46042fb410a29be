// The main RESCALE stage of the pixel-major tensor-core kernels (a thread holds 16 output columns of one pixel): the table of
// per-column constants in shared memory and the forms in which it is evaluated.
#ifndef MLEL_PIXEL_EPILOGUE_CUH
#define MLEL_PIXEL_EPILOGUE_CUH

#include <cstdint>

#include "device_common.cuh"

namespace mlel {
namespace tc {

// Constants of the main RESCALE stage for one output column, two shared-memory reads per element in the general form (see
// FastRescale): {mult, corr0, rnLo, rnHi, s2, bump} with the rounding constant for v < zpIn (input zero point folded in).
// Where wordsScaleApplies to every column and the corrections are small, one read: the WordsScale {low, high, mult, shift}
// with the correction folded in.  (The 64-bit addend first: as the middle of a 16-byte load, where no register pair starts, it
// was moved for every result.)
struct __align__(16) ColConst {
    int32_t mult;        // else WordsScale's low
    int32_t corr;        // correction of the most common border class; else WordsScale's high
    uint32_t rnLo, rnHi; // rounding constant; else WordsScale's mult and shift
    int32_t s2;          // max(shift - 32, 0)
    uint32_t bump;       // what the constant for v >= zpIn adds: 2^31 with double rounding and shift > 31, else 0
    int32_t s1;          // min(shift, 32)
    int32_t corr0;       // correction of the most common border class (what a border pixel swaps for its own)
};

enum : int { kGeneralForm = 0, kSignedWords = 1, kWords = 2 };

// The table's form where wordsScaleApplies to every column.
__device__ __forceinline__ int wordsForm(const DevRescale &m) { return wordsScaleSignFree(m.doubleRound != 0, m.outZp, m.lo) ? kWords : kSignedWords; }

__device__ __forceinline__ ColConst makeColConst(const FastRescale &f, int32_t corr0, const DevRescale &m, int form) {
    ColConst c;
    c.s1 = f.s1, c.s2 = f.s2, c.corr0 = corr0;
    c.bump = f.rpLo - f.rnLo; // (rp - rn) mod 2^32: 0 or 2^31
    if (form != kGeneralForm) {
        const int32_t x0 = int32_t(uint32_t(corr0) - uint32_t(f.zpIn));
        const WordsScale w = form == kWords ? makeWordsScale<false>(f.mult, f.s1 + f.s2, m.doubleRound != 0, x0, m.outZp)
                                            : makeWordsScale<true>(f.mult, f.s1 + f.s2, m.doubleRound != 0, x0, 0);
        c.mult = int32_t(w.low), c.corr = int32_t(w.high), c.rnLo = uint32_t(w.mult), c.rnHi = uint32_t(w.shift);
    } else {
        c.mult = f.mult, c.corr = corr0, c.rnLo = f.rnLo, c.rnHi = f.rnHi;
    }
    return c;
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

// 16 columns of one row by WordsScale, packed four results to a word.
template <bool SIGNED>
__device__ __forceinline__ void rescale16Words(const uint32_t (&acc)[16], uint32_t tabAddr, int32_t outZp, int32_t lo, int32_t hi,
                                               uint32_t (&packed)[4]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        int32_t y[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int j = 4 * q + e;
            uint32_t mult, low, high, shift;
            ldsV4(tabAddr + uint32_t(j) * 32u, low, high, mult, shift);
            const int32_t v = wordsScale<SIGNED>(WordsScale{int32_t(mult), int32_t(shift), low, high}, int32_t(acc[j]));
            y[e] = min(SIGNED ? __viaddmax_s32(v, outZp, lo) : max(v, lo), hi);
        }
        packed[q] = packSatS8(y[0], y[1], y[2], y[3]);
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
        packed[q] = packSatS8(y[0], y[1], y[2], y[3]);
    }
}

} // namespace tc
} // namespace mlel

#endif
