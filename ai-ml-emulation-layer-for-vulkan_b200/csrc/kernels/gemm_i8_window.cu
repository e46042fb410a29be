// int8 convolution windows on the tcgen05 tensor cores from one resident input tile (stride 1, at most 128 input channels).
//
// Why.  The im2col kernels fetch every tap of a tile's windows on its own: a 3x3 window moves each input pixel nine times
// from L2 into shared memory, and with few channels the copies, not the products, take the time: per 128 pixels of a
// 64-channel layer 9 x 192 rows of 128 bytes for 18 MMAs of some 50 cycles each.  Here a tile's input -- its pixels and
// the border its windows reach, zero-filled outside the image -- is fetched once, by one TMA box, and every tap's MMA reads
// it from another start address:
//
//   D[pixel, oc] = sum over taps (ky, kx) of X[pixel + ky * pitch + kx, :] * W[tap][oc, :]
//
// Pixels lie in shared memory `pitch` to an image row, a pixel's channels in 32, 64 or 128 bytes (the swizzle of that
// width).  A tensor-core operand is groups of eight consecutive rows a fixed stride apart, so two tile shapes work:
//   rows   - whole stretches of tileW pixels, the border columns included: operand row r is pixel r of the box (stride
//            8 pixels), rows that fall on border columns are computed and dropped;
//   blocks - 8 pixels wide and 16 high: group g is image row g (stride: one pitch).
// The host takes the shape with the least time by its count of tiles, copied rows and MMAs.
//
// Few channels (an RGB stem; stride 1 or 2).  A pixel of at most four channels is too small for an operand row (16 bytes at
// least).  A copy of the input gathers 16-byte units first -- four pixels of four (zero-padded) channels: at stride 1 the
// pixels x to x + 3 of a row, at stride 2 the 2 x 2 pixels under one output pixel -- so that an output pixel's window is
// whole units at constant distances and output pixels are one unit apart.  Rows of 16 bytes need no swizzle; an MMA takes
// two units per row, the second at its own distance (the descriptor's leading offset).  The loops are the same.
//
// The weights of a CTA's output channels (all taps) stay in shared memory for its lifetime; CTAs are persistent and take
// every (CTAs / channel tiles)-th pixel tile.  Warps 0-15 epilogue, 16 TMA, 17 MMA; accumulators alternate.
//
// Measured (3x3, im2col kernels before): 64 x 56 x 56, 64 -> 64 channels 37.2 -> 19.1 us, 32 -> 64 37.8 -> 15.5; 270 x 480,
// 96 -> 32 32.4 -> 11.9; 64 x 28 x 28, 128 -> 128 15.4 -> 13.8.  With the MMAs issued by a lane that their statement elects,
// 270 x 480, 96 -> 32 8.6 (not with few MMAs a tap and a long epilogue, see ummaLed).
// Bound now by the epilogue's RESCALEs and, with 128 channels, by the MMAs.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "gemm_i8_tcgen05.hpp"
#include "pixel_epilogue.cuh"
#include "tcgen05_common.cuh"

namespace mlel {
namespace {

using namespace tc;

constexpr int kWindowMaxStages = 4;
constexpr int kMaxUnitPairs = 8; // 32 bytes of window each: 7x7 at stride 2 has sixteen units, at stride 1 fourteen
constexpr size_t kWindowSmemLimit = 232448; // shared memory per CTA

// Geometry of a launch (see the head of the file).
struct WindowTiling {
    int32_t pixelBytes;   // bytes of one pixel in shared memory: 32, 64 or 128; of one unit: 16
    int32_t boxW, boxH;   // pixels of the box; boxW is the pitch
    int32_t tileW, tileH; // output pixels of a tile
    int32_t blocks;       // 1: 8 x 16 blocks, 0: rows
    int32_t stages, stageBytes;
    int32_t tilesX, tilesY, pixelTiles, channelTiles;
    int32_t originX, originY; // a window's first pixel (unit) minus the output pixel's own position
    int32_t weightBytes;      // of one channel tile
    int32_t unitsX, unitStep, unitPairs; // units: per window row, distance in a row, pairs of a window
    FastDiv divTilesX, divTilesY, divPitch;
};

struct __align__(8) WindowBarriers {
    uint64_t full[kWindowMaxStages], empty[kWindowMaxStages];
    uint64_t accFull[2], accEmpty[2];
    uint64_t weights;
    uint32_t tmemBase, forms;
};

// Descriptor of a K-major operand whose rows are `rowBytes` long in the swizzle of that width.
__device__ __forceinline__ uint64_t rowDesc(uint32_t addr, uint32_t rowBytes, uint32_t groupBytes) {
    const uint64_t layout = rowBytes == 128 ? 2 : (rowBytes == 64 ? 4 : 6);
    return (smemDesc(addr, 16, groupBytes) & ~(uint64_t(7) << 61)) | (layout << 61);
}

// Descriptor of a K-major operand without a swizzle: groups of eight 16-byte rows.
__device__ __forceinline__ uint64_t smemDescPlain(uint32_t addr, uint32_t leadingBytes, uint32_t groupBytes) {
    return smemDesc(addr, leadingBytes, groupBytes) & ~(uint64_t(7) << 61);
}

// One MMA by lane 0, named by a predicate and not elected: it takes 62 cycles to issue where an elected one takes 21 (see umma).
// That is the better pace for one or two MMAs a tap beside tiles of 64 channels, where most CTAs have two: their epilogue is the longer
// part, and MMAs that arrive no faster than the pipe takes them (50 cycles) leave the epilogue warps of that scheduler their issue slots.
// (us, elected and so: 16 x 56 x 56, 64 -> 64 7.8 and 7.4, 32 images 11.5 and 11.0, 64 -> 128 11.8 and 11.0, 8 x 61 x 19, 64 -> 464 9.9
// and 9.5, 270 x 480, 32 -> 64 10.8 and 10.2, 8 x 112 x 112, 32 -> 64 9.2 and 8.8.  A CTA's first tile has to wait for its MMAs: with one
// tile a CTA, 68 x 120, 64 -> 128, and with 1.8, 135 x 240, 32 -> 64, 0.1 us more.  Elsewhere the pace is the MMAs': 16 x 56 x 56, 64 -> 32
// 5.6 and 6.0, 96 -> 64 7.6 and 9.4, 270 x 480, 96 -> 32 8.6 and 11.4; tiles of 128 channels the same either way.)
__device__ __forceinline__ void ummaLed(uint32_t leader, uint32_t tmemD, DescWords a, DescWords b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p, l;\n\t.reg .b64 a, b;\n\t"
                 "setp.ne.b32 l, %8, 0;\n\t"
                 "setp.ne.b32 p, %6, 0;\n\t"
                 "mov.b64 a, {%1, %2};\n\t"
                 "mov.b64 b, {%3, %4};\n\t"
                 "@l tcgen05.mma.cta_group::1.kind::i8 [%0], a, b, %5, {%7, %7, %7, %7}, p;\n\t}"
                 ::"r"(tmemD), "r"(a.low), "r"(a.high), "r"(b.low), "r"(b.high), "r"(idesc), "r"(accumulate), "r"(0u), "r"(leader)
                 : "memory");
}

// ODD: output rows start at any address.  The warps that share 32 rows of the accumulator put them together in shared memory
// and store them as aligned words (storeRowBytes).  64 -> 63 channels, 8 x 56 x 56: 10.6 us on the pixel-major kernel, here
// 8.8; 30 x 30, 64 -> 65: 9.7 and 6.1.
template <int BN> constexpr int kOddPitch = BN + 4;                                        // bytes of a staged row
template <int BN> constexpr int kOddBytes = 4 * 32 * kOddPitch<BN> * (BN == 32 ? 2 : 1) + 16; // quarters x rows x sets

// BN: output channels of a tile (32, 64 or 128).  UNITS: the input is 16-byte units (see the head of the file).
// LED: for up to 64 input channels, 3x3 (see ummaLed).
template <int BN, bool UNITS, bool ODD, bool LED>
__global__ void __launch_bounds__(kThreadsTma, 1)
gemmI8Window(const __grid_constant__ CUtensorMap mapX, const __grid_constant__ CUtensorMap mapW, const GemmI8Params p,
             const WindowTiling g) {
    extern __shared__ uint8_t rawSmem[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(rawSmem) + 1023) & ~uintptr_t(1023));
    const int taps = p.KH * p.KW, tapBytes = BN * g.pixelBytes;
    uint8_t *weights = smem;
    uint8_t *stages = smem + g.weightBytes;
    ColConst *colTab = reinterpret_cast<ColConst *>(stages + g.stages * g.stageBytes);
    WindowBarriers *bars = reinterpret_cast<WindowBarriers *>(colTab + BN);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c0 = int(blockIdx.x % unsigned(g.channelTiles)) * BN;
    const int firstTile = int(blockIdx.x / unsigned(g.channelTiles)), tileStep = int(gridDim.x / unsigned(g.channelTiles));
    // warps that drain one accumulator: four per 16 columns; with 32 columns half of the warps take every other tile
    constexpr int kSets = BN == 32 ? 2 : 1, kGroups = 4 / kSets, kSteps = BN / 16 / kGroups;

    if (threadIdx.x == 0) {
        for (int s = 0; s < g.stages; ++s) {
            mbarInit(&bars->full[s], 1u);
            mbarInit(&bars->empty[s], 1u);
        }
        for (int b = 0; b < 2; ++b) {
            mbarInit(&bars->accFull[b], 1u);
            mbarInit(&bars->accEmpty[b], uint32_t(kEpilogueWarps / kSets));
        }
        mbarInit(&bars->weights, 1u);
        bars->forms = 1; // wordsScaleApplies to every column
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(&bars->tmemBase)),
                     "r"(uint32_t(2 * BN))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmemBase = bars->tmemBase;

    if (warp == kTmaWarp) {
        if (lane == 0) {
            // the weights are constants of the pipeline: before the launch ahead has finished
            mbarArriveExpectTx(&bars->weights, uint32_t(g.weightBytes));
            if (UNITS) {
                tmaLoad3d(&mapW, weights, &bars->weights, 0, c0, 0);
            } else {
                for (int t = 0; t < taps; ++t) {
                    tmaLoad3d(&mapW, weights + t * tapBytes, &bars->weights, 0, t, c0);
                }
            }
            dependencySync();
            int s = 0;
            uint32_t phase = 0;
            for (int tile = firstTile; tile < g.pixelTiles; tile += tileStep) {
                const uint32_t ty = fastDiv(uint32_t(tile), g.divTilesX), n = fastDiv(ty, g.divTilesY);
                const int x0 = (tile - int(ty) * g.tilesX) * g.tileW, y0 = int(ty - n * uint32_t(g.tilesY)) * g.tileH;
                if (!mbarWait(&bars->empty[s], phase ^ 1u, 91)) {
                    break;
                }
                mbarArriveExpectTx(&bars->full[s], uint32_t(g.boxW * g.boxH * g.pixelBytes));
                if (UNITS) { // (a unit is two elements of the map)
                    tmaLoad3d(&mapX, stages + s * g.stageBytes, &bars->full[s], 2 * (x0 + g.originX), y0 + g.originY, int(n));
                } else {
                    tmaLoad4d(&mapX, stages + s * g.stageBytes, &bars->full[s], 0, x0 + g.originX, y0 + g.originY, int(n));
                }
                if (++s == g.stages) {
                    s = 0;
                    phase ^= 1u;
                }
            }
        }
        __syncwarp();
    } else if (warp == kMmaWarp) {
        // The whole warp runs the loop and one lane issues: with nothing divergent around them the descriptors stay in uniform
        // registers.  (With the loop inside `if (lane == 0)` every MMA cost the thread some 200 cycles of moves and waits behind
        // the epilogue warps of its scheduler, 4000 of a 64-channel tile's 4600.)  A wait that runs out only ends the waiting:
        // the later MMAs read old bytes, the recorded error tells.
        dependencySync();
        constexpr uint32_t idesc = instrDesc(BN, false);
        const uint32_t groupBytes = uint32_t((g.blocks ? g.boxW : 8) * g.pixelBytes), leader = lane == 0 ? 1u : 0u;
        const uint64_t descX = rowDesc(smemAddr(stages), uint32_t(g.pixelBytes), groupBytes);
        const uint64_t descW = rowDesc(smemAddr(weights), uint32_t(g.pixelBytes), uint32_t(8 * g.pixelBytes));
        const uint32_t lowX = uint32_t(descX), highX = uint32_t(descX >> 32), lowW = uint32_t(descW), highW = uint32_t(descW >> 32);
        const uint32_t tapStep = uint32_t(p.dilX * g.pixelBytes) >> 4, rowStep = uint32_t(p.dilY * g.boxW * g.pixelBytes) >> 4,
                       weightStep = uint32_t(tapBytes) >> 4, stageStep = uint32_t(g.stageBytes) >> 4;
        const int windowH = p.KH, windowW = p.KW, pixelTiles = g.pixelTiles, stageCount = g.stages;
        // UNITS: first words of the descriptors of every pair's MMA, from the stage's and the weights' start
        uint32_t pairX[kMaxUnitPairs], pairHigh = 0, weightHigh = 0;
        if (UNITS) {
            const auto unitAt = [&](int u) { return uint32_t(u / g.unitsX * g.boxW + u % g.unitsX * g.unitStep); };
#pragma unroll
            for (int m = 0; m < kMaxUnitPairs; ++m) {
                const bool last = 2 * m + 1 >= g.unitsX * windowH; // an odd unit out: any second one, its weights are zero
                pairX[m] = unitAt(2 * m) + ((last ? 1u : unitAt(2 * m + 1) - unitAt(2 * m)) << 16);
            }
            pairHigh = uint32_t(smemDescPlain(0, 0, groupBytes) >> 32), weightHigh = uint32_t(smemDescPlain(0, 0, 128) >> 32);
        }
        // slices: MMAs per tap, 32 channels each; three: a 3x3 window, unrolled
        const auto tiles = [&](auto sliceCount, auto three) {
            constexpr int kSlices = decltype(sliceCount)::value;
            constexpr bool kThree = decltype(three)::value;
            bool failed = !mbarWait(&bars->weights, 0u, 92);
            int s = 0;
            uint32_t phase = 0, tileCount = 0, stageX = lowX;
            for (int tile = firstTile; tile < pixelTiles; tile += tileStep, ++tileCount) {
                const uint32_t buf = tileCount & 1u;
                failed = failed || !mbarWait(&bars->accEmpty[buf], ((tileCount >> 1) & 1u) ^ 1u, 93) || !mbarWait(&bars->full[s], phase, 94);
                __syncwarp();
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t tmemD = tmemBase + buf * uint32_t(BN);
                const auto tap = [&](uint32_t x, uint32_t w, bool first) {
                    if constexpr (LED) {
                        ummaLed(leader, tmemD, {x, highX}, {w, highW}, idesc, first ? 0u : 1u);
                        if (kSlices == 2) {
                            ummaLed(leader, tmemD, {x + 2u, highX}, {w + 2u, highW}, idesc, 1u);
                        }
                    } else {
                        ummaBlock(tmemD, {x, highX}, 2, {w, highW}, 2, idesc, first ? 0u : 1u, kSlices);
                    }
                };
                if (UNITS) {
                    const uint32_t stage = smemAddr(stages + s * g.stageBytes) >> 4, w = (smemAddr(weights) >> 4) + (uint32_t(BN) << 16);
#pragma unroll
                    for (int m = 0; m < kMaxUnitPairs; ++m) {
                        if (m < g.unitPairs) {
                            umma(tmemD, {stage + pairX[m], pairHigh}, {w + uint32_t(2 * m * BN), weightHigh}, idesc, m == 0 ? 0u : 1u);
                        }
                    }
                } else if (kThree && kSlices == 1 && !LED) { // (a window row to a statement)
#pragma unroll
                    for (int ky = 0; ky < 3; ++ky) {
                        ummaBlock(tmemD, {stageX + uint32_t(ky) * rowStep, highX}, tapStep, {lowW + uint32_t(3 * ky) * weightStep, highW},
                                  weightStep, idesc, ky == 0 ? 0u : 1u, 3);
                    }
                } else if (kThree) {
#pragma unroll
                    for (int t = 0; t < 9; ++t) {
                        tap(stageX + uint32_t(t / 3) * rowStep + uint32_t(t % 3) * tapStep, lowW + uint32_t(t) * weightStep, t == 0);
                    }
                } else {
                    uint32_t w = lowW, rowX = stageX;
                    for (int ky = 0; ky < windowH; ++ky, rowX += rowStep) {
                        uint32_t x = rowX;
                        for (int kx = 0; kx < windowW; ++kx, x += tapStep, w += weightStep) {
                            tap(x, w, ky + kx == 0);
                        }
                    }
                }
                ummaCommit(&bars->empty[s]);
                ummaCommit(&bars->accFull[buf]);
                stageX += stageStep;
                if (++s == stageCount) {
                    s = 0;
                    stageX = lowX;
                    phase ^= 1u;
                }
            }
        };
        const bool three = windowH == 3 && windowW == 3;
        if constexpr (UNITS) {
            tiles(std::integral_constant<int, 1>{}, std::false_type{});
        } else if constexpr (LED) {
            p.IC <= 32 ? tiles(std::integral_constant<int, 1>{}, std::true_type{}) : tiles(std::integral_constant<int, 2>{}, std::true_type{});
        } else {
            using Three = std::true_type;
            using Any = std::false_type;
            switch ((p.IC + UMMA_K - 1) / UMMA_K) {
            case 1:
                three ? tiles(std::integral_constant<int, 1>{}, Three{}) : tiles(std::integral_constant<int, 1>{}, Any{});
                break;
            case 2:
                three ? tiles(std::integral_constant<int, 2>{}, Three{}) : tiles(std::integral_constant<int, 2>{}, Any{});
                break;
            case 3:
                three ? tiles(std::integral_constant<int, 3>{}, Three{}) : tiles(std::integral_constant<int, 3>{}, Any{});
                break;
            default:
                three ? tiles(std::integral_constant<int, 4>{}, Three{}) : tiles(std::integral_constant<int, 4>{}, Any{});
            }
        }
    } else {
        // ---- epilogue: the table of this CTA's channels, then a tile row (pixel) per lane, 16 columns per step
        const int32_t zpMain = p.epi.main.inZp, outZp = p.epi.main.outZp, lo = p.epi.main.lo, hi = p.epi.main.hi;
        const bool twoRounds = p.epi.main.doubleRound != 0;
        FastRescale f{};
        int32_t corr0 = 0;
        if (threadIdx.x < BN) {
            const int col = c0 + int(threadIdx.x), ci = (p.epi.main.perChannel && col < p.N) ? col : 0;
            f = makeFastRescale(__ldg(p.epi.main.mult + ci), int32_t(__ldg(p.epi.main.shift + ci)), zpMain, twoRounds);
            if (!wordsScaleApplies(f.mult, f.s1 + f.s2, twoRounds)) {
                atomicAnd(&bars->forms, 0u);
            }
            corr0 = col < p.N ? __ldg(p.corr + int64_t(p.baseClass) * p.N + col) : 0;
        }
        epilogueSync();
        const uint32_t holds = *const_cast<volatile uint32_t *>(&bars->forms);
        const int form = holds != 0 && p.corrSmall != 0 ? wordsForm(p.epi.main) : kGeneralForm;
        if (threadIdx.x < BN) {
            colTab[threadIdx.x] = makeColConst(f, corr0, p.epi.main, form);
        }
        epilogueSync();
        dependencySync();

        const int quarter = warp & 3, part = warp >> 2, set = part / kGroups, group = part - set * kGroups;
        const int row = quarter * 32 + lane;
        const int yy = g.blocks ? row >> 3 : int(fastDiv(uint32_t(row), g.divPitch)), xx = g.blocks ? row & 7 : row - yy * g.boxW;
        const bool rowInTile = yy < g.tileH && xx < g.tileW;
        const uint32_t tabAddr = smemAddr(colTab);
        uint32_t tileCount = 0;
        bool failed = false;
        // ODD: this quarter's (and set's) rows, after the barriers
        const uint32_t staged = ((smemAddr(bars) + uint32_t(sizeof(WindowBarriers)) + 15u) & ~15u) + uint32_t((quarter + 4 * set) * 32 * kOddPitch<BN>);
        const auto meet = [&] { asm volatile("bar.sync %0, %1;" ::"r"(2 + quarter + 4 * set), "r"(kGroups * 32) : "memory"); };
        for (int tile = firstTile; tile < g.pixelTiles; tile += tileStep, ++tileCount) {
            const uint32_t buf = tileCount & 1u;
            if (kSets == 2 && int(buf) != set) {
                continue;
            }
            const uint32_t ty = fastDiv(uint32_t(tile), g.divTilesX), n = fastDiv(ty, g.divTilesY);
            const int x = (tile - int(ty) * g.tilesX) * g.tileW + xx, y = int(ty - n * uint32_t(g.tilesY)) * g.tileH + yy;
            const bool valid = rowInTile && x < p.OW && y < p.OH;
            int cls = p.baseClass;
            if (p.rowClass != nullptr && valid) {
                cls = int(__ldg(p.rowClass + y)) * p.numColClasses + int(__ldg(p.colClass + x));
            }
            int8_t *dst = p.out8 + ((int64_t(n) * p.OH + y) * p.OW + x) * p.ldOut + c0;
            if (ODD) { // after a wait that ran out the warp still meets the others
                failed = failed || !mbarWait(&bars->accFull[buf], (tileCount >> 1) & 1u, 95);
            } else if (!mbarWait(&bars->accFull[buf], (tileCount >> 1) & 1u, 95)) {
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t taddr = tmemBase + buf * uint32_t(BN) + (uint32_t(quarter * 32) << 16);
#pragma unroll 1
            for (int st = 0; st < kSteps; ++st) {
                const int cl = (group * kSteps + st) * 16;
                uint32_t acc[16];
                tmemLoad16(taddr + uint32_t(cl), acc);
                tmemWait16(acc);
                if (st == kSteps - 1) {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    if (lane == 0) {
                        mbarArrive(&bars->accEmpty[buf]);
                    }
                }
                if (!valid || c0 + cl >= p.N) {
                    continue;
                }
                if (cls != p.baseClass) {
                    // a pixel whose window crosses the border: swap the table's correction for its own class's
                    if (ODD) {
                        const int32_t *own = p.corr + int64_t(cls) * p.N + c0 + cl;
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            if (c0 + cl + j < p.N) {
                                acc[j] += uint32_t(__ldg(own + j)) - uint32_t(colTab[cl + j].corr0);
                            }
                        }
                    }
                    const int4 *own = reinterpret_cast<const int4 *>(p.corr + int64_t(cls) * p.N + c0 + cl);
#pragma unroll
                    for (int q = 0; q < (ODD ? 0 : 4); ++q) {
                        const int4 v = __ldg(own + q);
                        acc[4 * q] += uint32_t(v.x) - uint32_t(colTab[cl + 4 * q].corr0);
                        acc[4 * q + 1] += uint32_t(v.y) - uint32_t(colTab[cl + 4 * q + 1].corr0);
                        acc[4 * q + 2] += uint32_t(v.z) - uint32_t(colTab[cl + 4 * q + 2].corr0);
                        acc[4 * q + 3] += uint32_t(v.w) - uint32_t(colTab[cl + 4 * q + 3].corr0);
                    }
                }
                uint32_t packed[4];
                const uint32_t tab = tabAddr + uint32_t(cl) * 32u;
                if (form == kWords) {
                    rescale16Words<false>(acc, tab, outZp, lo, hi, packed);
                } else if (form == kSignedWords) {
                    rescale16Words<true>(acc, tab, outZp, lo, hi, packed);
                } else {
                    rescale16General(acc, tab, zpMain, outZp, lo, hi, packed);
                }
                if (ODD) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        asm volatile("st.shared.u32 [%0], %1;" ::"r"(staged + uint32_t(lane * kOddPitch<BN> + cl + 4 * q)), "r"(packed[q]) : "memory");
                    }
                    continue;
                }
                *reinterpret_cast<int4 *>(dst + cl) = make_int4(int(packed[0]), int(packed[1]), int(packed[2]), int(packed[3]));
            }
            if (ODD) {
                meet();
                const uint32_t live = __ballot_sync(0xffffffffu, valid);
                const int length = min(BN, p.N - c0);
#pragma unroll 2
                for (int r = group; r < 32; r += kGroups) {
                    int8_t *to = reinterpret_cast<int8_t *>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(dst), r));
                    if ((live >> r) & 1u) {
                        storeRowBytes(to, staged + uint32_t(r * kOddPitch<BN>), length, lane);
                    }
                }
                meet(); // before the next tile's rows
            }
        }
    }
    __syncthreads();
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmemBase), "r"(uint32_t(2 * BN)) : "memory");
    }
}

// ---- host side --------------------------------------------------------------------------------------------

// CTAs of a channel tile.
int windowCtas(const WindowTiling &g) { return std::max(1, std::min(smCount() / g.channelTiles, g.pixelTiles)); }

template <int BN, bool UNITS, bool ODD, bool LED = false>
int launchWindowRows(const CUtensorMap &mapX, const CUtensorMap &mapW, const GemmI8Params &p, const WindowTiling &g, size_t smem,
                 cudaStream_t s) {
    auto kernel = gemmI8Window<BN, UNITS, ODD, LED>;
    if (!allowDynamicSmem(reinterpret_cast<const void *>(kernel), kWindowSmemLimit)) {
        return MLEL_ERROR_DEVICE;
    }
    const int perChannelTile = windowCtas(g);
    const cudaError_t err = launchOverlapped(kernel, perChannelTile * g.channelTiles, kThreadsTma, smem, s, mapX, mapW, p, g);
    if (err != cudaSuccess) {
        setLastError(std::string("int8 window launch: ") + cudaGetErrorString(err));
        return MLEL_ERROR_DEVICE;
    }
    return MLEL_SUCCESS;
}

// Output rows that do not all start on 16-byte boundaries.
bool windowOddRows(const GemmI8Params &p) { return p.ldOut % 16 != 0 || (reinterpret_cast<uintptr_t>(p.out8) & 15u) != 0; }

template <int BN, bool UNITS>
int launchWindow(const CUtensorMap &mapX, const CUtensorMap &mapW, const GemmI8Params &p, const WindowTiling &g, size_t smem,
                 cudaStream_t s) {
    if (windowOddRows(p)) {
        return launchWindowRows<BN, UNITS, true>(mapX, mapW, p, g, smem, s);
    }
    if constexpr (BN == 64 && !UNITS) {
        if (p.IC <= 64 && p.KH == 3 && p.KW == 3 && 15 * int64_t(windowCtas(g)) <= 8 * int64_t(g.pixelTiles)) {
            return launchWindowRows<BN, UNITS, false, true>(mapX, mapW, p, g, smem, s);
        }
    }
    return launchWindowRows<BN, UNITS, false>(mapX, mapW, p, g, smem, s);
}

size_t windowSmem(const WindowTiling &g, int bn, bool odd) {
    return 1024 + size_t(g.weightBytes) + size_t(g.stages) * g.stageBytes + size_t(bn) * sizeof(ColConst) + sizeof(WindowBarriers) +
           (odd ? size_t(bn == 32 ? kOddBytes<32> : (bn == 64 ? kOddBytes<64> : kOddBytes<128>)) : 0);
}

// What a tiling is chosen for: the reach of a window past its first pixel (unit) and the work of a tile.
struct WindowShape {
    int reachX, reachY;
    int pixelBytes;
    int weightRowBytes; // weights of one output channel
    int mmas;           // per tile
    int boxLimitW;
};

// Tiling of p with output tiles of bn channels; false: it does not fit.  *cost: estimated cycles of a CTA (the slowest of
// MMAs, copies and epilogue per tile, times the tiles of the busiest CTA).
bool windowTiling(const GemmI8Params &p, const WindowShape &w, int bn, WindowTiling *best, double *cost) {
    const int images = p.M / (p.OH * p.OW);
    bool found = false;
    const auto consider = [&](bool blocks, int tileW, int tileH) {
        WindowTiling g{};
        g.pixelBytes = w.pixelBytes;
        g.weightBytes = w.weightRowBytes * bn;
        g.blocks = blocks ? 1 : 0;
        g.tileW = tileW, g.tileH = tileH;
        g.boxW = tileW + w.reachX, g.boxH = tileH + w.reachY;
        if (g.boxW > w.boxLimitW || g.boxH > 256) {
            return;
        }
        // pixels that the MMAs of the last tap read (rows of the operand past the box hold old bytes; their results are dropped)
        const int reach = w.reachY * g.boxW + w.reachX + (blocks ? 15 * g.boxW + 8 : 128) + (w.pixelBytes == 16 ? 1 : 0);
        g.stageBytes = (std::max(reach, g.boxW * g.boxH) * g.pixelBytes + 1023) / 1024 * 1024;
        g.stages = kWindowMaxStages;
        while (g.stages > 1 && windowSmem(g, bn, windowOddRows(p)) > kWindowSmemLimit) {
            --g.stages;
        }
        if (g.stages < 2) {
            return;
        }
        g.tilesX = (p.OW + tileW - 1) / tileW, g.tilesY = (p.OH + tileH - 1) / tileH;
        const int64_t tiles = int64_t(images) * g.tilesX * g.tilesY;
        if (tiles >= (int64_t(1) << 30)) {
            return;
        }
        g.pixelTiles = int(tiles);
        g.channelTiles = (p.N + bn - 1) / bn;
        const int ctas = smCount() / g.channelTiles;
        if (ctas < 1) {
            return;
        }
        const double mma = double(w.mmas) * (32 + bn / 4), copy = double(g.boxW) * g.boxH * g.pixelBytes / 50,
                     epilogue = 13.0 * std::min(bn, p.N);
        const double cycles = (std::max(mma, std::max(copy, epilogue)) + 150) * double((g.pixelTiles + ctas - 1) / ctas);
        if (!found || cycles < *cost) {
            found = true;
            *cost = cycles;
            *best = g;
        }
    };
    consider(true, 8, 16);
    for (int pieces = 1; pieces <= 16; ++pieces) { // rows: the image row in equal pieces, as many of them as 128 operand rows hold
        const int tileW = (p.OW + pieces - 1) / pieces;
        if (tileW > 128) {
            continue;
        }
        const int tileH = std::min(p.OH, (128 - tileW) / (tileW + w.reachX) + 1);
        consider(false, tileW, tileH);
        if (tileW < 16) {
            break;
        }
    }
    return found;
}

// The tile width and tiling of least estimated time; 0: none fits.
int chooseTiling(const GemmI8Params &p, const WindowShape &w, WindowTiling *g) {
    int bn = 0;
    double cost = 0;
    for (const int width : {32, 64, 128}) {
        WindowTiling t{};
        double c = 0;
        if ((width == 32 || width < 2 * p.N) && windowTiling(p, w, width, &t, &c) && (bn == 0 || c < cost)) {
            bn = width, *g = t, cost = c;
        }
    }
    g->divTilesX = makeFastDiv(g->tilesX), g->divTilesY = makeFastDiv(g->tilesY), g->divPitch = makeFastDiv(g->boxW);
    return bn;
}

// Packed tensor (dims[0] fastest), elements of one byte or of eight.
template <int RANK>
bool makeWindowMap(CUtensorMap *map, uint64_t kind, const void *base, const cuuint64_t (&dims)[RANK], const cuuint32_t (&box)[RANK],
                   bool wide = false) {
    EncodeTiledFn fn = encodeTiled();
    if (fn == nullptr) {
        return false;
    }
    cuuint64_t strides[RANK - 1];
    cuuint32_t elemStrides[RANK];
    MapKey key{{kind, reinterpret_cast<uint64_t>(base)}};
    for (int i = 0; i < RANK; ++i) {
        if (i + 1 < RANK) {
            strides[i] = (i == 0 ? (wide ? 8 : 1) : strides[i - 1]) * dims[i];
        }
        elemStrides[i] = 1;
        key.v[2 + i] = dims[i], key.v[8 + i] = box[i];
    }
    const CUtensorMapSwizzle swizzle =
        wide || box[0] < 32 ? CU_TENSOR_MAP_SWIZZLE_NONE
        : box[0] == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : (box[0] == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
    return rememberedMap(map, key, [&](CUtensorMap *m) {
        return fn(m, wide ? CU_TENSOR_MAP_DATA_TYPE_UINT64 : CU_TENSOR_MAP_DATA_TYPE_UINT8, RANK, const_cast<void *>(base), dims, strides, box, elemStrides,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    });
}

} // namespace

// Stride 1 because the tensor core walks pixels at a constant distance; at most 128 channels because a CTA keeps the weights
// of all taps (and a pixel is one swizzled row); more than one tap because a 1x1 window is fetched once anyway.
bool gemmI8WindowApplies(const GemmI8Problem &q) {
    const GemmI8Params &p = q.params;
    const int mode = tensorCoreTuning().windowKernel.load(std::memory_order_relaxed);
    return mode != 0 && p.out8 != nullptr && p.epi.hasMain && !p.epi.hasResidual && q.aMatrix == nullptr && !q.bMnMajor && q.batches == 1 &&
           p.gatherTable == nullptr && p.strideX == 1 && p.strideY == 1 && p.IC % 16 == 0 && p.IC <= 128 && p.KH * p.KW > 1 && p.padLeft >= 0 && p.padTop >= 0 &&
           ((reinterpret_cast<uintptr_t>(p.in) | reinterpret_cast<uintptr_t>(q.bMatrix) | reinterpret_cast<uintptr_t>(p.corr)) & 15u) == 0;
}

int gemmI8WindowLaunch(const GemmI8Problem &q, cudaStream_t s, bool *taken) {
    GemmI8Params p = q.params;
    *taken = false;
    const int taps = p.KH * p.KW, pixelBytes = p.IC <= 32 ? 32 : (p.IC <= 64 ? 64 : 128);
    const WindowShape w{(p.KW - 1) * p.dilX, (p.KH - 1) * p.dilY, pixelBytes, taps * pixelBytes, taps * ((p.IC + 31) / 32), 256};
    WindowTiling g{};
    const int bn = chooseTiling(p, w, &g);
    if (bn == 0) {
        return MLEL_SUCCESS;
    }
    g.originX = -p.padLeft, g.originY = -p.padTop;
    const int images = p.M / (p.OH * p.OW);
    CUtensorMap mapX{}, mapW{};
    const cuuint64_t xDims[4] = {cuuint64_t(p.IC), cuuint64_t(p.W), cuuint64_t(p.H), cuuint64_t(images)};
    const cuuint32_t xBox[4] = {cuuint32_t(g.pixelBytes), cuuint32_t(g.boxW), cuuint32_t(g.boxH), 1};
    const cuuint64_t wDims[3] = {cuuint64_t(p.IC), cuuint64_t(taps), cuuint64_t(p.N)};
    const cuuint32_t wBox[3] = {cuuint32_t(g.pixelBytes), 1, cuuint32_t(bn)};
    if (!makeWindowMap(&mapX, 5, p.in, xDims, xBox) || !makeWindowMap(&mapW, 6, q.bMatrix, wDims, wBox)) {
        return MLEL_SUCCESS; // another kernel fetches the taps one by one
    }
    *taken = true;
    g_tensorCoreLaunches[4].fetch_add(1, std::memory_order_relaxed);
    const size_t smem = windowSmem(g, bn, windowOddRows(p));
    return bn == 32   ? launchWindow<32, false>(mapX, mapW, p, g, smem, s)
           : bn == 64 ? launchWindow<64, false>(mapX, mapW, p, g, smem, s)
                      : launchWindow<128, false>(mapX, mapW, p, g, smem, s);
}

int gemmI8UnitsLaunch(const GemmI8Problem &q, const UnitWindow &u, cudaStream_t s) {
    GemmI8Params p = q.params;
    p.KH = u.unitRows; // (rows of units)
    const int units = (u.unitsX * u.unitRows + 1) / 2 * 2;
    const WindowShape w{(u.unitsX - 1) * u.unitStep, u.unitRows - 1, 16, units * 16, units / 2, 128};
    WindowTiling g{};
    const int bn = chooseTiling(p, w, &g);
    if (bn == 0 || units > 2 * kMaxUnitPairs) {
        setLastError("int8 window of few channels: no tiling");
        return MLEL_ERROR_UNKNOWN;
    }
    g.originX = u.originX, g.originY = u.originY;
    g.unitsX = u.unitsX, g.unitStep = u.unitStep, g.unitPairs = units / 2;
    CUtensorMap mapX{}, mapW{};
    const cuuint64_t xDims[3] = {cuuint64_t(2) * u.width, cuuint64_t(u.height), cuuint64_t(p.M / (p.OH * p.OW))};
    const cuuint32_t xBox[3] = {cuuint32_t(2 * g.boxW), cuuint32_t(g.boxH), 1};
    const cuuint64_t wDims[3] = {16, cuuint64_t(p.N), cuuint64_t(units)};
    const cuuint32_t wBox[3] = {16, cuuint32_t(bn), cuuint32_t(units)};
    if (!makeWindowMap(&mapX, 7, u.units, xDims, xBox, true) || !makeWindowMap(&mapW, 8, q.bMatrix, wDims, wBox)) {
        setLastError("int8 window of few channels: no tensor map");
        return MLEL_ERROR_DEVICE;
    }
    g_tensorCoreLaunches[4].fetch_add(1, std::memory_order_relaxed);
    const size_t smem = windowSmem(g, bn, windowOddRows(p));
    return bn == 32   ? launchWindow<32, true>(mapX, mapW, p, g, smem, s)
           : bn == 64 ? launchWindow<64, true>(mapX, mapW, p, g, smem, s)
                      : launchWindow<128, true>(mapX, mapW, p, g, smem, s);
}

int windowErrorWord() { return readErrorWord(); }

} // namespace mlel
