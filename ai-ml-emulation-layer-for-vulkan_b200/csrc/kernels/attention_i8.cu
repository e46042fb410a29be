// Quantised attention as one kernel: score product, row-wise softmax and context product of an int8 transformer layer
// without the [batch, queries, keys] tensors in memory.
//
// The operators it stands for (GraphPipeline::fuseAttention) and their shaders:
//   S = MATMUL(Q, K^T)                                        int32   matmul.comp:30-73
//   U = RESCALE(S - REDUCE_MAX(S))                            int16   reduce.comp, elementwise_binary.comp, rescale.comp
//   E = TABLE(U);  D = TABLE(RESCALE(REDUCE_SUM(E)))          int32   table.comp:17-52
//   P = RESCALE(MUL(E, D, shift))                             int8    mul.comp:24-59, rescale.comp
//   C = RESCALE(MATMUL(P, V))                                 int8
// with the head split and merge (TRANSPOSE, transpose.comp) absorbed as strides of Q, K, V and C.  Every step is the
// operator's own integer arithmetic, so the result is the same bits.
//
// Why.  As kernels of their own the steps move the int32 score tensor five times: at 32 sequences of 384 tokens and 12
// heads that is 226 MB a pass and 294 us of a 525 us layer.  Here a block takes 128 queries of one head: the scores of
// up to 512 keys fit its tensor memory (a lane per query, a column per key), the exponentials replace them there, the
// probabilities go to shared memory as the next product's A operand, and only Q, K, V and C touch memory: 57 us, and no
// row length, odd ones included, leaves the tensor cores (3 sequences of 197 tokens: 640 -> 12 us a layer).
//
// What bounds it: the integer arithmetic of the softmax, about 15 instructions per score (two RESCALEs, a table
// look-up with interpolation, a 64-bit product); the two products take under a tenth of that.  Hence
//   * each element-wise RESCALE is one 32 x 32 + 64 bit multiply-add, whose high word is shifted: the operands' signs are
//     known, so the double-rounding terms are constants, and the row maximum and both zero points are part of the addend;
//   * a table entry holds (value, step to the next value) as two int16, so that one look-up and one two-way dot product
//     give value * 128 + step * fraction;
//   * P is stored minus its zero point, as unsigned bytes, so that the second product needs no correction row;
//   * packing saturates (cvt.pack.sat), which is the clamp of the last RESCALE.
// Sixteen warps share the 128 x keys scores (four per quarter of the tensor-memory lanes, 32-column slices in turn) and
// exchange row maxima and row sums through shared memory.  Up to 192 keys a block has eight of them, so that two blocks
// fit an SM and one's products run under the other's softmax.  One more warp feeds them: its first lane issues the TMA
// loads and the MMAs.  Where scores and context fit tensor memory side by side it issues the next tile's score product
// as soon as the probabilities of this one are out; while that runs the softmax warps store the previous tile's context
// rows, and this tile's context product follows under the next softmax.  Otherwise the two products take turns.
// Clock stamps of a tile of 384 keys, 15 200 cycles before this order: 1200 waiting for scores, 700 row maximum, 2400
// context rows (most of it waiting for their product), 6200 exponentials, 400 at the barrier, 4000 probabilities.
//
// Of the integer pipes the multiply-add one counts: a 32 x 32 -> 64 bit product takes it four cycles a warp, a 32-bit one
// two.  A RESCALE whose multiplier is a small number times a power of two (powers of two are the usual scales inside a
// quantised softmax) has its constants divided by that power on the host where everything then fits 32 bits (NARROW).
#include <algorithm>

#include "attention_i8.hpp"
#include "tcgen05_common.cuh"

namespace mlel {

namespace {

using namespace tc;

constexpr int kTokenBox = 32;  // tokens per TMA load
constexpr int kRowBytes = 128; // a SWIZZLE_128B row: one query or key, up to 128 bytes of head dimension

struct AttentionParams {
    int8_t *out;
    int32_t Sq, Sk, d, keysPad; // keysPad: keys rounded up to the 32 of an MMA's K step
    uint32_t tiles;
    FastDiv queryTiles, heads;
    int32_t contextColumn; // first tensor-memory column of the context; 0: it takes the columns of the scores
    int64_t oStride[3];    // bytes: sequence, head, token
    const int16_t *expTable, *recipTable;
    AttentionPlan plan;
};

struct AttentionShared {
    uint64_t loadedQK, loadedV;        // TMA
    uint64_t scoresDone, contextDone;  // MMA
    uint64_t probsReady, contextRead;  // softmax warps
    uint32_t tmemBase;
};

// dp2a: c + lo16(a) * byte0(b) + hi16(a) * byte1(b), a signed, b unsigned
__device__ __forceinline__ int32_t dp2aLow(uint32_t a, uint32_t b, int32_t c) {
    int32_t r;
    asm("dp2a.lo.s32.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}
// bytes (sat(y1) << 8 | sat(y0)) below the low half of `upper`
template <bool UNSIGNED> __device__ __forceinline__ uint32_t packSat(int32_t y1, int32_t y0, uint32_t upper) {
    uint32_t r;
    if (UNSIGNED) {
        asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(y1), "r"(y0), "r"(upper));
    } else {
        asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(y1), "r"(y0), "r"(upper));
    }
    return r;
}
__device__ __forceinline__ uint32_t ldsU32(uint32_t addr) {
    uint32_t v;
    asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr)); // written before the first tile, never again
    return v;
}
constexpr int kSlice = 32; // score columns a warp takes at a time
// (load and wait in one statement: the registers reach no other instruction in between)
__device__ __forceinline__ void tmemRead32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmemStore32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
                 "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
                 "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
                 "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                 "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
                 "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
                 "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
                 : "memory");
}

// 4-D tensor map {head dimension, token, head, sequence} over an int8 operand with a box of 32 tokens by one 128-byte
// SWIZZLE_128B row: bytes past the head dimension and tokens past the last arrive as zeros.
__device__ __forceinline__ void loadTokens(const CUtensorMap *map, uint8_t *dst, uint64_t *bar, int first, int count, int head,
                                           int sequence) {
    for (int r = 0; r < count; r += kTokenBox) {
        tmaLoad4d(map, dst + r * kRowBytes, bar, 0, first + r, head, sequence);
    }
}

// (x * mult + addend) >> 32 + shift from the 64-bit product, or >> shift from the 32-bit one.
template <bool NARROW>
__device__ __forceinline__ int32_t scaleKnownSign(int32_t x, int32_t mult, int64_t addend, int32_t shift) {
    if (NARROW) {
        return (x * mult + int32_t(addend)) >> shift;
    }
    return int32_t((int64_t(x) * int64_t(mult) + addend) >> 32) >> shift;
}

template <int WARPS, bool UNSIGNED_P, bool NARROW>
__global__ void __launch_bounds__(WARPS * 32 + 32, WARPS == 8 ? 2 : 1)
attentionI8Kernel(const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapK,
                  const __grid_constant__ CUtensorMap mapV, const __grid_constant__ AttentionParams p) {
    constexpr int kThreads = WARPS * 32 + 32;
    constexpr int kGroups = WARPS / 4; // softmax warps per quarter of the tensor-memory lanes
    extern __shared__ uint8_t rawSmem[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(rawSmem) + 1023) & ~uintptr_t(1023));
    uint8_t *tileQ = smem;
    uint8_t *tileK = tileQ + BM * kRowBytes;
    uint8_t *tileV = tileK + p.keysPad * kRowBytes;
    uint8_t *tileP = tileV + p.keysPad * kRowBytes; // 128 keys per 16 KB block, K-major
    const int blocksP = (p.keysPad + 127) / 128;
    uint32_t *expLut = reinterpret_cast<uint32_t *>(tileP + blocksP * (BM * BK)); // 512 x (value << 16 | step)
    int32_t *partMax = reinterpret_cast<int32_t *>(expLut + 512);                 // [kGroups][128]
    int32_t *partSum = partMax + kGroups * BM;
    AttentionShared *shared = reinterpret_cast<AttentionShared *>(partSum + kGroups * BM);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int quarter = warp & 3, columnGroup = warp >> 2;
    const int row = quarter * 32 + lane; // query inside the tile = tensor-memory lane
    const bool sideBySide = p.contextColumn != 0;
    uint32_t columns = 32;
    while (columns < uint32_t(max(p.keysPad, p.contextColumn + p.d))) {
        columns *= 2;
    }

    if (threadIdx.x == 0) {
        mbarInit(&shared->loadedQK, 1);
        mbarInit(&shared->loadedV, 1);
        mbarInit(&shared->scoresDone, 1);
        mbarInit(&shared->contextDone, 1);
        mbarInit(&shared->probsReady, WARPS);
        mbarInit(&shared->contextRead, WARPS);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = threadIdx.x; i < 512; i += kThreads) {
        const int32_t value = p.expTable[i], next = p.expTable[i + 1];
        expLut[i] = (uint32_t(value) << 16) | (uint32_t(next - value) & 0xffffu); // the step fits int16 (fuseAttention)
    }
    if (warp == WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(&shared->tmemBase)),
                     "r"(columns)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmemBase = shared->tmemBase;
    dependencySync(); // from here on activations are read and written

    struct Tile {
        uint32_t n, h;
        int q0;
    };
    const auto tileOf = [&](uint32_t t) {
        const uint32_t b = fastDiv(t, p.queryTiles), n = fastDiv(b, p.heads);
        return Tile{n, b - n * p.heads.d, int(t - b * p.queryTiles.d) * BM};
    };

    if (warp == WARPS) {
        {
            // ---------------- loads (by one lane) and MMAs (by the whole warp, see ummaBlockPeek) ----------------
            const auto loadQK = [&](const Tile &t) {
                if (lane == 0) {
                    mbarArriveExpectTx(&shared->loadedQK, uint32_t((BM + p.keysPad) * kRowBytes));
                    loadTokens(&mapQ, tileQ, &shared->loadedQK, t.q0, BM, int(t.h), int(t.n));
                    loadTokens(&mapK, tileK, &shared->loadedQK, 0, p.keysPad, int(t.h), int(t.n));
                }
                __syncwarp();
            };
            const auto loadV = [&](const Tile &t) {
                if (lane == 0) {
                    mbarArriveExpectTx(&shared->loadedV, uint32_t(p.keysPad * kRowBytes));
                    loadTokens(&mapV, tileV, &shared->loadedV, 0, p.keysPad, int(t.h), int(t.n));
                }
                __syncwarp();
            };
            const auto wait = [&](uint64_t *bar, uint32_t parity, int code) { return mbarWaitWarp(bar, parity, code); };
            const DescWords descQ = descWords(smemDesc(smemAddr(tileQ), 16, 1024)), descK = descWords(smemDesc(smemAddr(tileK), 16, 1024));
            const DescWords descP = descWords(smemDesc(smemAddr(tileP), 16, 1024)), descV = descWords(smemDesc(smemAddr(tileV), BK * 128, 1024));
            const auto scoreProduct = [&] {
                for (int n0 = 0; n0 < p.keysPad; n0 += 256) {
                    const int n = min(256, p.keysPad - n0);
                    for (int ks = 0; ks * UMMA_K < p.d; ++ks) {
                        umma(tmemBase + uint32_t(n0), {descQ.low + uint32_t(2 * ks), descQ.high},
                             {descK.low + uint32_t(n0 * (kRowBytes >> 4) + 2 * ks), descK.high}, instrDesc(n, false), ks > 0 ? 1u : 0u);
                    }
                }
                ummaCommit(&shared->scoresDone);
            };
            const auto contextProduct = [&] {
                // A format 0: unsigned 8-bit
                const uint32_t idesc = instrDesc(p.d, true) & (UNSIGNED_P ? ~(7u << 7) : ~0u);
                for (int ks = 0; ks * UMMA_K < p.keysPad; ++ks) {
                    umma(tmemBase + uint32_t(p.contextColumn), {descP.low + uint32_t((ks >> 2) * ((BM * BK) >> 4) + 2 * (ks & 3)), descP.high},
                         {descV.low + uint32_t(ks * ((UMMA_K * kRowBytes) >> 4)), descV.high}, idesc, ks > 0 ? 1u : 0u);
                }
                ummaCommit(&shared->contextDone);
            };
            uint32_t t = blockIdx.x;
            bool ok = true;
            if (t < p.tiles) {
                loadQK(tileOf(t));
                loadV(tileOf(t));
                ok = wait(&shared->loadedQK, 0, 71);
                if (ok) {
                    scoreProduct();
                }
            }
            for (uint32_t i = 0; t < p.tiles && ok; ++i, t += gridDim.x) {
                const uint32_t parity = i & 1u;
                const uint32_t next = t + gridDim.x;
                const bool more = next < p.tiles;
                ok = wait(&shared->scoresDone, parity, 72); // Q and K have been read
                if (ok && more) {
                    loadQK(tileOf(next));
                }
                ok = ok && wait(&shared->probsReady, parity, 73) && wait(&shared->loadedV, parity, 74) &&
                     (!more || wait(&shared->loadedQK, parity ^ 1u, 71));
                if (!ok) {
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (sideBySide && more) {
                    scoreProduct();
                }
                if (sideBySide && i > 0) { // the previous tile's context has been stored
                    ok = wait(&shared->contextRead, parity ^ 1u, 76);
                    if (!ok) {
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                }
                contextProduct();
                ok = wait(&shared->contextDone, parity, 75); // V and the probabilities have been read
                if (ok && more) {
                    loadV(tileOf(next));
                }
                if (!sideBySide && more) {
                    ok = ok && wait(&shared->contextRead, parity, 76);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (ok) {
                        scoreProduct();
                    }
                }
            }
        }
        __syncwarp();
    } else {
    // ---------------- softmax and context rows ----------------
    // the warps of one quarter, i.e. of the same 32 rows
    const auto quarterSync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(1 + quarter), "n"(kGroups * 32) : "memory"); };
    const AttentionPlan &a = p.plan;
    const int slices = p.keysPad / kSlice;
    const uint32_t lutAddr = smemAddr(expLut);
    const uint32_t laneAddr = tmemBase + (uint32_t(quarter * 32) << 16);
    const auto contextRows = [&](const Tile &tile) {
        int8_t *dst = p.out + tile.n * p.oStride[0] + tile.h * p.oStride[1] + int64_t(tile.q0 + row) * p.oStride[2];
        for (int c = columnGroup; 16 * c < p.d; c += kGroups) {
            uint32_t s[16];
            tmemLoad16(laneAddr + uint32_t(p.contextColumn + 16 * c), s);
            tmemWait16(s);
            uint32_t packed[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                uint32_t w = 0;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    w |= uint32_t(uint8_t(fastRescale(a.context, int32_t(s[4 * q + j]), a.contextOutZp, -128, 127)))
                         << (8 * j);
                }
                packed[q] = w;
            }
            if (tile.q0 + row < p.Sq) {
                *reinterpret_cast<uint4 *>(dst + 16 * c) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
            }
        }
    };

    // Waits as a warp.  After a wait that ran out the warp keeps to the barriers of its quarter and does nothing else.
    const auto waitAll = [](uint64_t *bar, uint32_t phase, int code) {
        const bool done = mbarWaitWarp(bar, phase, code);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        return done;
    };
    bool ok = true;
    uint32_t i = 0;
    Tile last{};
    for (uint32_t t = blockIdx.x; t < p.tiles; t += gridDim.x, ++i) {
        const uint32_t parity = i & 1u;
        ok = ok && waitAll(&shared->scoresDone, parity, 77);

        // ---- row maximum
        int32_t top = int32_t(0x80000000u);
        for (int c = ok ? columnGroup : slices; c < slices; c += kGroups) {
            uint32_t s[kSlice];
            tmemRead32(laneAddr + uint32_t(kSlice * c), s);
            const int live = p.Sk - kSlice * c; // columns of real keys in this slice
            if (live < kSlice) {
#pragma unroll
                for (int j = 0; j < kSlice; ++j) {
                    s[j] = j < live ? s[j] : 0x80000000u;
                }
            }
#pragma unroll
            for (int j = 0; j < kSlice; j += 2) {
                top = __vimax3_s32(top, int32_t(s[j]), int32_t(s[j + 1]));
            }
        }
        partMax[columnGroup * BM + row] = top;
        quarterSync();
#pragma unroll
        for (int g = 0; g < kGroups; ++g) {
            top = max(top, partMax[g * BM + row]);
        }

        // ---- exponentials, in place; row sum
        // (s - top) * mult + addend as s * mult + (addend - top * mult)
        const int64_t diffAddend = a.diffAddend - int64_t(top) * int64_t(a.diffMult); // NARROW: inside 32 bits
        uint32_t sum = 0;
        for (int c = ok ? columnGroup : slices; c < slices; c += kGroups) {
            uint32_t s[kSlice];
            tmemRead32(laneAddr + uint32_t(kSlice * c), s);
            const int live = p.Sk - kSlice * c;
            if (live < kSlice) { // columns of padding: any score up to the maximum
#pragma unroll
                for (int j = 0; j < kSlice; ++j) {
                    s[j] = j < live ? s[j] : uint32_t(top);
                }
            }
#pragma unroll
            for (int j = 0; j < kSlice; ++j) {
                // int16 result + 32768
                const uint32_t u = uint32_t(max(scaleKnownSign<NARROW>(int32_t(s[j]), a.diffMult, diffAddend, a.diffShift), 0));
                s[j] = uint32_t(dp2aLow(ldsU32(lutAddr + (u >> 7) * a.entryBytes), (u & 0x7fu) | a.unitByte, 0));
            }
            if (live < kSlice) {
#pragma unroll
                for (int j = 0; j < kSlice; ++j) {
                    s[j] = j < live ? s[j] : 0u;
                }
            }
#pragma unroll
            for (int j = 0; j < kSlice; j += 2) {
                sum += s[j] + s[j + 1];
            }
            tmemStore32(laneAddr + uint32_t(kSlice * c), s);
        }
        partSum[columnGroup * BM + row] = int32_t(sum);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        quarterSync();
        sum = 0;
#pragma unroll
        for (int g = 0; g < kGroups; ++g) {
            sum += uint32_t(partSum[g * BM + row]);
        }
        int32_t recip;
        {
            const int32_t u = fastRescale(a.denom, int32_t(sum), a.denomOutZp, -32768, 32767);
            const int32_t index = (u + 32768) >> 7, base = __ldg(p.recipTable + index), next = __ldg(p.recipTable + index + 1);
            recip = int32_t((uint32_t(base) << 7) + uint32_t(next - base) * uint32_t(u & 0x7f));
        }

        // ---- probabilities minus their zero point, into the A operand of the context product
        if (sideBySide && i > 0) { // which the previous tile's product has read
            ok = ok && waitAll(&shared->contextDone, parity ^ 1u, 78);
        }
        for (int c = ok ? columnGroup : slices; c < slices; c += kGroups) {
            uint32_t s[kSlice];
            tmemRead32(laneAddr + uint32_t(kSlice * c), s);
            uint32_t packed[kSlice / 4];
#pragma unroll
            for (int q = 0; q < kSlice / 4; ++q) {
                int32_t y[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint64_t prod = uint64_t(int64_t(int32_t(s[4 * q + j])) * int64_t(recip)) + uint64_t(a.mulRound);
                    const int32_t x = int32_t(__funnelshift_r(uint32_t(prod), uint32_t(prod >> 32), uint32_t(a.mulShift)));
                    y[j] = scaleKnownSign<NARROW>(x, a.probMult, a.probAddend, a.probShift);
                }
                packed[q] = packSat<UNSIGNED_P>(y[1], y[0], packSat<UNSIGNED_P>(y[3], y[2], 0u));
            }
            // 16-byte pieces 2 (c & 3) and the next of this row in the 128-key block c >> 2
            const uint32_t dst = smemAddr(tileP) + uint32_t((c >> 2) * (BM * BK) + row * BK);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + uint32_t(((2 * (c & 3) + h) ^ (row & 7)) << 4)),
                             "r"(packed[4 * h]), "r"(packed[4 * h + 1]), "r"(packed[4 * h + 2]), "r"(packed[4 * h + 3])
                             : "memory");
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // the tensor core reads the probabilities
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0 && ok) {
            mbarArrive(&shared->probsReady);
        }
        // The context in tensor memory: the previous tile's while the next scores are made, or, where it takes columns
        // of the scores, this tile's before they are.
        const Tile tile = tileOf(t);
        if (!sideBySide) {
            last = tile;
            ok = ok && waitAll(&shared->contextDone, parity, 79);
        }
        if (!sideBySide || i > 0) {
            if (ok) {
                contextRows(last);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0 && ok) {
                mbarArrive(&shared->contextRead);
            }
        }
        last = tile;
    }
    if (sideBySide && i > 0 && ok && waitAll(&shared->contextDone, (i - 1u) & 1u, 78)) {
        contextRows(last);
    }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == WARPS) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmemBase), "r"(columns) : "memory");
    }
}

size_t attentionSmem(int keysPad, int warps) {
    return 1024 + size_t(BM) * kRowBytes + 2 * size_t(keysPad) * kRowBytes + size_t((keysPad + 127) / 128) * BM * BK + 512 * 4 +
           2 * size_t(warps / 4) * BM * 4 + sizeof(AttentionShared);
}

bool makeTokenMap(CUtensorMap *map, const void *base, int d, int tokens, int heads, int sequences, const int64_t (&stride)[3]) {
    EncodeTiledFn fn = encodeTiled();
    if (fn == nullptr) {
        setLastError("cuTensorMapEncodeTiled is not available from the driver");
        return false;
    }
    const cuuint64_t dims[4] = {cuuint64_t(d), cuuint64_t(tokens), cuuint64_t(heads), cuuint64_t(sequences)};
    const cuuint64_t strides[3] = {cuuint64_t(stride[2]), cuuint64_t(stride[1]), cuuint64_t(stride[0])};
    const cuuint32_t box[4] = {kRowBytes, kTokenBox, 1, 1};
    const cuuint32_t elemStrides[4] = {1, 1, 1, 1};
    const MapKey key{{4, reinterpret_cast<uint64_t>(base), uint64_t(d), uint64_t(tokens), uint64_t(heads), uint64_t(sequences),
                      uint64_t(stride[0]), uint64_t(stride[1]), uint64_t(stride[2])}};
    return rememberedMap(map, key, [&](CUtensorMap *m) {
        const CUresult rc = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<void *>(base), dims, strides, box, elemStrides,
                               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (rc != CUDA_SUCCESS) {
            setLastError("attention: cuTensorMapEncodeTiled failed with code " + std::to_string(int(rc)));
            return false;
        }
        return true;
    });
}

template <int WARPS>
int launchAttention(const CUtensorMap (&maps)[3], AttentionParams p, cudaStream_t s) {
    const size_t smem = attentionSmem(p.keysPad, WARPS);
    const bool narrow = p.plan.narrow;
    auto kernel = p.plan.unsignedProb
                      ? (narrow ? attentionI8Kernel<WARPS, true, true> : attentionI8Kernel<WARPS, true, false>)
                      : (narrow ? attentionI8Kernel<WARPS, false, true> : attentionI8Kernel<WARPS, false, false>);
    if (!allowDynamicSmem(reinterpret_cast<const void *>(kernel),
                          attentionSmem(WARPS == 8 ? kAttentionTwoBlockKeys : kAttentionMaxKeys, WARPS))) {
        return MLEL_ERROR_DEVICE;
    }
    const int blocksPerSm = WARPS == 8 ? 2 : 1;
    p.contextColumn = p.keysPad + p.d <= 512 / blocksPerSm ? p.keysPad : 0;
    const int grid = int(std::min<int64_t>(p.tiles, int64_t(smCount()) * blocksPerSm));
    if (launchOverlapped(kernel, grid, WARPS * 32 + 32, smem, s, maps[0], maps[1], maps[2], p) != cudaSuccess) {
        setLastError(std::string("attention: ") + cudaGetErrorString(cudaGetLastError()));
        return MLEL_ERROR_DEVICE;
    }
    return MLEL_SUCCESS;
}

} // namespace

int attentionErrorWord() { return readErrorWord(); }

int attentionFused(const AttentionPlan &plan, const TView &q, const TView &k, const TView &v, const TView &expTable,
                   const TView &recipTable, const TView &out, cudaStream_t s) {
    if (((reinterpret_cast<uintptr_t>(q.ptr) | reinterpret_cast<uintptr_t>(k.ptr) | reinterpret_cast<uintptr_t>(v.ptr) |
          reinterpret_cast<uintptr_t>(out.ptr)) & 15u) != 0) {
        setLastError("attention: operands must be 16-byte aligned");
        return MLEL_ERROR_UNKNOWN;
    }
    AttentionParams p{};
    p.plan = plan;
    p.out = reinterpret_cast<int8_t *>(out.ptr);
    p.expTable = reinterpret_cast<const int16_t *>(expTable.ptr);
    p.recipTable = reinterpret_cast<const int16_t *>(recipTable.ptr);
    p.Sq = plan.queries, p.Sk = plan.keys, p.d = plan.headDim;
    p.keysPad = (p.Sk + 31) / 32 * 32;
    const int64_t queryTiles = (p.Sq + BM - 1) / BM;
    p.tiles = uint32_t(queryTiles * plan.batches);
    p.queryTiles = makeFastDiv(queryTiles);
    p.heads = makeFastDiv(plan.heads);
    for (int i = 0; i < 3; ++i) {
        p.oStride[i] = plan.oStride[i];
    }
    CUtensorMap maps[3];
    const int sequences = plan.batches / plan.heads;
    if (!makeTokenMap(&maps[0], q.ptr + plan.qOffset, p.d, p.Sq, plan.heads, sequences, plan.qStride) ||
        !makeTokenMap(&maps[1], k.ptr + plan.kOffset, p.d, p.Sk, plan.heads, sequences, plan.kStride) ||
        !makeTokenMap(&maps[2], v.ptr + plan.vOffset, p.d, p.Sk, plan.heads, sequences, plan.vStride)) {
        return MLEL_ERROR_DEVICE;
    }
    return p.keysPad <= kAttentionTwoBlockKeys ? launchAttention<8>(maps, p, s)
                                              : launchAttention<16>(maps, p, s);
}

} // namespace mlel
