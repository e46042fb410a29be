// Residual add with layer norm of a quantised transformer as one register-resident kernel: the row program
//   t = RESCALE(a) + RESCALE(b);  c = t - MUL(SUM(t), k1, s1);  d = TABLE(RESCALE(MUL(SUM(MUL(c, c, s2)), k2, s3)))
//   out = RESCALE(MUL(c, d, s4))
// on int8 rows (reduce.comp, elementwise_binary.comp, mul.comp, rescale.comp, table.comp).  rowMachine() hands a program
// over when rowNormMatch() recognises it: these instructions in this order, operands of ADD and MUL either way round.
// Anything else (a gain or bias per channel) runs in the row machine or as kernels of its own.  The row machine keeps every
// value of a row in shared memory and pays its interpreter and a shared-memory round trip per operator: 63 us for 12 288
// rows of 768, where the bytes (28 MB, mostly in L2) take about 5.
//
// A warp owns a row and keeps it in registers, four neighbouring elements per lane and 128-element group.  What is left
// is bound by the integer instructions of the arithmetic.  NARROW: RESCALEs whose multiplier is a small number times a
// power of two are divided by that power on the host (the scales of a fixed-point normalisation are powers of two), and
// squares that fit 32 bits stay there: a 32 x 32 -> 64 bit product costs the multiply-add pipe twice a 32-bit one.
// Otherwise the same steps run on the 64-bit forms.  Measured (events around one launch): 63 -> 18 us.
//
// SHORT: where moreover both inputs are scaled up by whole numbers and the output is scaled down by a power of two -- a
// residual stream in int8 whose normalisation keeps fractional bits --, an element is some ten instructions instead of thirty:
//   * RESCALE(a) + RESCALE(b) is one two-way dot product of the byte pair with the two multipliers;
//   * the last MUL and RESCALE, floor((floor((c * d + r) / 2^s) + e) / 2^u), are one: floor((c * d + r + e * 2^s) / 2^(s + u)),
//     and with d shifted left by 32 - s - u, once a row, the result is the high word of one 64-bit multiply-add;
//   * what double rounding adds depends on the sign of c * d + r, i.e. on which side of one number per row c lies;
//   * packing saturates.
// (12 288 rows of 768 in a replayed encoder: 15.6 -> 11.0 us behind the attention, 21.6 -> 15.7 behind the FFN; 3 x 197 tokens, four layers, 201 -> 189.5.)
#include <string>

#include "device_common.cuh"
#include "kernels.hpp"
#include "launch_overlapped.cuh"

namespace mlel {

namespace {

// floor((x * mult + add -+ bump) / 2^shift) on 32 bits: add holds +bump, which x < zpIn turns into -bump.
struct SlimScale {
    int32_t mult, add, shift, bump, zpIn;
};
struct NormScale {
    FastRescale full;
    SlimScale slim;
    int32_t outZp, lo, hi;
};
struct NormParams {
    const int8_t *a, *b;
    int8_t *out;
    const int16_t *table;
    int64_t rows;
    int32_t len;
    NormScale scaleA, scaleB, scaleVar, scaleOut;
    int32_t meanMult, meanShift, squareShift, varMult, varShift, normShift;
    // SHORT
    int32_t pairMult, pairAdd; // multipliers of a (low half) and b; what both RESCALEs add
    int32_t factorShift;
    int64_t outAdd;  // addend of the output's multiply-add for a negative product
    uint32_t outBump; // what a product that is not negative adds to it (no carry into the high word)
};

__device__ __forceinline__ int32_t mulShifted(int32_t x, int32_t y, int32_t shift) {
    int64_t p = int64_t(x) * int64_t(y);
    if (shift > 0) {
        p = int64_t(uint64_t(p) + (1ull << (shift - 1))) >> shift;
    }
    return int32_t(uint32_t(uint64_t(p)));
}
template <bool NARROW, bool SIGNED> __device__ __forceinline__ int32_t scaled(const NormScale &s, int32_t x) {
    if (NARROW) {
        int32_t v = x * s.slim.mult + s.slim.add;
        if (SIGNED) {
            v -= x < s.slim.zpIn ? 2 * s.slim.bump : 0;
        }
        return (v >> s.slim.shift) + s.outZp;
    }
    return fastRescale(s.full, x, s.outZp, s.lo, s.hi);
}

enum : int { kWideForm = 0, kNarrowForm = 1, kShortForm = 2 };

// GROUPS x 128 elements a row at most.
template <int GROUPS, int FORM>
__global__ void __launch_bounds__(256) rowNormKernel(const __grid_constant__ NormParams p) {
    constexpr bool NARROW = FORM != kWideForm;
    dependencySync();
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t(gridDim.x) * blockDim.x) >> 5;
    for (int64_t row = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; row < p.rows; row += warps) {
        const int8_t *a = p.a + row * p.len, *b = p.b + row * p.len;
        // (read once: marked so, 0.24 us less of 12 288 rows of 768 than ordinary loads)
        uint32_t wa[GROUPS], wb[GROUPS];
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) {
            const int i = g * 128 + lane * 4;
            wa[g] = i < p.len ? __ldcs(reinterpret_cast<const uint32_t *>(a + i)) : 0u;
            wb[g] = i < p.len ? __ldcs(reinterpret_cast<const uint32_t *>(b + i)) : 0u;
        }
        int32_t t[GROUPS][4];
        uint32_t sum = 0;
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) {
            const bool live = g * 128 + lane * 4 < p.len;
            if (FORM == kShortForm) {
                const int32_t low = int32_t(__byte_perm(wa[g], wb[g], 0x5140)), high = int32_t(__byte_perm(wa[g], wb[g], 0x7362));
                t[g][0] = __dp2a_lo(p.pairMult, low, p.pairAdd), t[g][1] = __dp2a_hi(p.pairMult, low, p.pairAdd);
                t[g][2] = __dp2a_lo(p.pairMult, high, p.pairAdd), t[g][3] = __dp2a_hi(p.pairMult, high, p.pairAdd);
                if (live) {
                    sum += uint32_t(t[g][0]) + uint32_t(t[g][1]) + uint32_t(t[g][2]) + uint32_t(t[g][3]);
                }
                continue;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                t[g][k] = int32_t(uint32_t(scaled<NARROW, false>(p.scaleA, int32_t(int8_t(wa[g] >> (8 * k))))) +
                                  uint32_t(scaled<NARROW, false>(p.scaleB, int32_t(int8_t(wb[g] >> (8 * k))))));
                sum += live ? uint32_t(t[g][k]) : 0u;
            }
        }
        sum = __reduce_add_sync(0xffffffffu, sum);
        const int32_t mean = mulShifted(int32_t(sum), p.meanMult, p.meanShift);
        uint32_t squares = 0;
        const int32_t squareRound = p.squareShift > 0 ? 1 << (p.squareShift - 1) : 0;
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) {
            const bool live = g * 128 + lane * 4 < p.len;
            uint32_t q[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int32_t c = int32_t(uint32_t(t[g][k]) - uint32_t(mean));
                t[g][k] = c;
                q[k] = uint32_t(NARROW ? (c * c + squareRound) >> p.squareShift : mulShifted(c, c, p.squareShift));
            }
            if (live) {
                squares += q[0] + q[1] + q[2] + q[3];
            }
        }
        squares = __reduce_add_sync(0xffffffffu, squares);
        const int32_t var = fastRescale(p.scaleVar.full, mulShifted(int32_t(squares), p.varMult, p.varShift), p.scaleVar.outZp,
                                        p.scaleVar.lo, p.scaleVar.hi); // an int16 value
        const int32_t index = (var + 32768) >> 7, base = __ldg(p.table + index), next = __ldg(p.table + index + 1);
        const int32_t factor = int32_t((uint32_t(base) << 7) + uint32_t(next - base) * uint32_t(var & 0x7f));
        int8_t *out = p.out + row * p.len;
        // SHORT: c above `edge` adds `above` to the low word, else `below`
        int32_t edge = 0, scaledFactor = 0;
        uint32_t above = 0, below = 0;
        if (FORM == kShortForm) {
            scaledFactor = int32_t(uint32_t(factor) << p.factorShift);
            const uint32_t size = uint32_t(abs(factor)), round = 1u << (p.normShift - 1);
            const int32_t reach = size > round ? 0 : (size != 0 ? int32_t(round / size) : 1 << 30); // c * factor >= -round up to here
            const uint32_t low = uint32_t(uint64_t(p.outAdd));
            edge = factor < 0 ? reach : -reach - 1;
            above = factor < 0 ? low : low + p.outBump;
            below = factor < 0 ? low + p.outBump : low;
        }
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) {
            uint32_t word = 0;
            if (FORM == kShortForm) {
                int32_t y[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint64_t addend = (uint64_t(p.outAdd) & ~uint64_t(0xffffffffu)) | uint64_t(t[g][k] > edge ? above : below);
                    y[k] = int32_t((uint64_t(int64_t(t[g][k]) * int64_t(scaledFactor)) + addend) >> 32);
                }
                word = packSatS8(y[0], y[1], y[2], y[3]);
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    int32_t x;
                    if (NARROW) { // 1 <= normShift <= 31
                        const uint64_t prod = uint64_t(int64_t(t[g][k]) * int64_t(factor)) + (1ull << (p.normShift - 1));
                        x = int32_t(__funnelshift_r(uint32_t(prod), uint32_t(prod >> 32), uint32_t(p.normShift)));
                    } else {
                        x = mulShifted(t[g][k], factor, p.normShift);
                    }
                    int32_t r = scaled<NARROW, true>(p.scaleOut, x);
                    r = min(max(r, p.scaleOut.lo), p.scaleOut.hi);
                    word |= uint32_t(uint8_t(r)) << (8 * k);
                }
            }
            const int i = g * 128 + lane * 4;
            if (i < p.len) {
                *reinterpret_cast<uint32_t *>(out + i) = word;
            }
        }
    }
}

// RESCALE parameters {mult, shift, inZp, outZp, lo, hi, doubleRound} for operands of at most xMax in size.  Returns
// whether the 32-bit form holds; *bound is then the largest result in size.  signedAllowed: the kernel evaluates the
// sign term of double rounding.
bool makeNormScale(const int32_t (&q)[7], int64_t xMax, bool signedAllowed, NormScale *s, int64_t *bound) {
    s->full = makeFastRescale(q[0], q[1], q[2], q[6] != 0);
    s->outZp = q[3], s->lo = q[4], s->hi = q[5];
    const int shift = q[1];
    const bool bumped = q[6] != 0 && shift > 31;
    if (shift < 0 || shift > 62 || q[0] < 0 || (bumped && !signedAllowed)) {
        return false;
    }
    // divide multiplier, rounding term and double-rounding term by the power of two they share
    int64_t m = q[0], round = shift > 0 ? int64_t(1) << (shift - 1) : 0, bump = bumped ? int64_t(1) << 30 : 0;
    int k = 0;
    while (k < shift && ((m | bump) & 1) == 0 && (k + 1 == shift || (round & 1) == 0)) {
        m >>= 1, bump >>= 1, round >>= 1; // at k + 1 == shift the rounding term is below one unit and falls away
        ++k;
    }
    const int64_t reach = xMax + 2 * std::abs(int64_t(q[2]));
    if (reach >= (int64_t(1) << 31)) {
        return false; // (the product below would leave 64 bits)
    }
    const int64_t most = reach * m + round + 2 * bump;
    if (shift - k > 31 || most >= (int64_t(1) << 31)) {
        return false;
    }
    s->slim = SlimScale{int32_t(m), int32_t(round + bump - int64_t(q[2]) * m), shift - k, int32_t(bump), q[2]};
    *bound = (most >> (shift - k)) + 1 + std::abs(int64_t(q[3]));
    return *bound < (int64_t(1) << 31);
}

} // namespace

bool rowNormMatch(const RowProgram &program) {
    static constexpr int kOps[16] = {ROW_LOAD, ROW_RESCALE, ROW_LOAD,       ROW_RESCALE, ROW_ADD,     ROW_REDUCE_SUM, ROW_MUL, ROW_SUB,
                                     ROW_MUL,  ROW_REDUCE_SUM, ROW_MUL, ROW_RESCALE, ROW_TABLE16, ROW_MUL,        ROW_RESCALE, ROW_STORE};
    if (program.insts.size() != 16 || program.len % 4 != 0 || program.len > 2048) {
        return false;
    }
    // which instruction's result every slot and per-row word holds, and what each instruction reads
    int full[64], value[kMaxRowValues];
    int a[16], b[16];
    for (int n = 0; n < 16; ++n) {
        const RowInst &in = program.insts[size_t(n)];
        if (in.op != kOps[n]) {
            return false;
        }
        const auto source = [&](const RowOperand &o) {
            return o.kind == ROW_FULL && o.index < 64 ? full[o.index] : (o.kind == ROW_VALUE ? value[o.index] : -1);
        };
        a[n] = source(in.a), b[n] = source(in.b);
        if (in.dst.kind == ROW_FULL) {
            if (in.dst.index >= 64) {
                return false;
            }
            full[in.dst.index] = n;
        } else if (in.dst.kind == ROW_VALUE) {
            value[in.dst.index] = n;
        }
    }
    const auto &in = program.insts;
    const auto immediate = [&](int n, int operand) { // MUL of a per-row value with a constant, in either order
        return (a[n] == operand && in[size_t(n)].b.kind == ROW_IMMEDIATE) || (b[n] == operand && in[size_t(n)].a.kind == ROW_IMMEDIATE);
    };
    return in[0].dtype == MLEL_I8 && in[2].dtype == MLEL_I8 && in[15].dtype == MLEL_I8 && in[0].dst.kind == ROW_FULL &&
           in[2].dst.kind == ROW_FULL && a[1] == 0 && a[3] == 2 && ((a[4] == 1 && b[4] == 3) || (a[4] == 3 && b[4] == 1)) &&
           a[5] == 4 && immediate(6, 5) && a[7] == 4 && b[7] == 6 && a[8] == 7 && b[8] == 7 && a[9] == 8 && immediate(10, 9) &&
           a[11] == 10 && a[12] == 11 && ((a[13] == 7 && b[13] == 12) || (a[13] == 12 && b[13] == 7)) && a[14] == 13 &&
           a[15] == 14;
}

int rowNorm(const RowProgram &program, const TView *T, cudaStream_t s) {
    const auto &in = program.insts;
    NormParams p{};
    p.a = reinterpret_cast<const int8_t *>(T[in[0].tensor].ptr);
    p.b = reinterpret_cast<const int8_t *>(T[in[2].tensor].ptr);
    p.out = reinterpret_cast<int8_t *>(T[in[15].tensor].ptr);
    p.table = reinterpret_cast<const int16_t *>(T[in[12].tensor].ptr);
    p.rows = program.rows;
    p.len = program.len;
    const auto constantOf = [&](int n) { return in[size_t(n)].a.kind == ROW_IMMEDIATE ? in[size_t(n)].a.imm : in[size_t(n)].b.imm; };
    p.meanMult = constantOf(6), p.meanShift = in[6].p[0];
    p.squareShift = in[8].p[0];
    p.varMult = constantOf(10), p.varShift = in[10].p[0];
    p.normShift = in[13].p[0];
    // Bounds from int8 operands through every step; a table value times 128 is below 2^22 in size.
    int64_t boundA = 0, boundB = 0, unused = 0;
    bool narrow = makeNormScale(in[1].p, 128, false, &p.scaleA, &boundA);
    narrow = makeNormScale(in[3].p, 128, false, &p.scaleB, &boundB) && narrow;
    makeNormScale(in[11].p, 0, true, &p.scaleVar, &unused);
    int64_t xMax = int64_t(1) << 40;
    if (narrow && p.normShift >= 1 && p.normShift <= 31 && p.squareShift <= 30) {
        const int64_t t = boundA + boundB, total = t * p.len;
        narrow = total < (int64_t(1) << 31);
        const int64_t mean = narrow ? ((total * std::abs(int64_t(p.meanMult))) >> p.meanShift) + 1 : 0, c = t + mean;
        narrow = narrow && c < 46000 && c * c + (int64_t(1) << p.squareShift) < (int64_t(1) << 31);
        xMax = ((c << 22) >> p.normShift) + 1;
    } else {
        narrow = false;
    }
    narrow = makeNormScale(in[14].p, narrow ? xMax : 0, true, &p.scaleOut, &unused) && narrow;
    // SHORT (see the head of the file).  |c| < 2^16 and |factor| <= 2^22, so c * factor * 2^factorShift stays below 2^46.
    const SlimScale &sa = p.scaleA.slim, &sb = p.scaleB.slim, &so = p.scaleOut.slim;
    bool shortForm = narrow && sa.shift == 0 && sb.shift == 0 && sa.mult <= 32767 && sb.mult <= 32767 && so.mult == 1 && so.zpIn == 0 &&
                     p.scaleOut.lo <= -128 && p.scaleOut.hi >= 127;
    if (shortForm) {
        const int shift = p.normShift + so.shift;
        p.factorShift = 32 - shift;
        shortForm = shift >= 24 && shift <= 32;
        if (shortForm) {
            p.pairMult = int32_t((uint32_t(sb.mult) << 16) | uint32_t(sa.mult));
            p.pairAdd = int32_t(uint32_t(sa.add) + uint32_t(p.scaleA.outZp) + uint32_t(sb.add) + uint32_t(p.scaleB.outZp));
            // rounding of the MUL; that of the RESCALE less both double-rounding terms; output zero point
            const int64_t add = (int64_t(1) << (p.normShift - 1)) + (int64_t(so.add - 2 * so.bump) * (int64_t(1) << p.normShift)) +
                                int64_t(p.scaleOut.outZp) * (int64_t(1) << shift);
            const uint64_t bump = uint64_t(2 * int64_t(so.bump)) << (p.normShift + p.factorShift);
            p.outAdd = add * (int64_t(1) << p.factorShift);
            p.outBump = uint32_t(bump);
            shortForm = (uint64_t(uint32_t(uint64_t(p.outAdd))) + bump) < (uint64_t(1) << 32);
        }
    }

    const int groups = (p.len + 127) / 128;
    const int grid = gridFor(p.rows * 32, 256, 16);
    const auto launch = [&](auto brief, auto slim, auto full) {
        launchOverlapped(shortForm ? brief : (narrow ? slim : full), grid, 256, 0, s, p);
    };
    if (groups <= 2) {
        launch(rowNormKernel<2, kShortForm>, rowNormKernel<2, kNarrowForm>, rowNormKernel<2, kWideForm>);
    } else if (groups <= 4) {
        launch(rowNormKernel<4, kShortForm>, rowNormKernel<4, kNarrowForm>, rowNormKernel<4, kWideForm>);
    } else if (groups <= 6) {
        launch(rowNormKernel<6, kShortForm>, rowNormKernel<6, kNarrowForm>, rowNormKernel<6, kWideForm>);
    } else if (groups <= 8) {
        launch(rowNormKernel<8, kShortForm>, rowNormKernel<8, kNarrowForm>, rowNormKernel<8, kWideForm>);
    } else {
        launch(rowNormKernel<16, kShortForm>, rowNormKernel<16, kNarrowForm>, rowNormKernel<16, kWideForm>);
    }
    const cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) {
        setLastError(std::string("fused layer norm: ") + cudaGetErrorString(err));
        return MLEL_ERROR_DEVICE;
    }
    return MLEL_SUCCESS;
}

} // namespace mlel
