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
// probabilities go to shared memory as the next product's A operand, and only Q, K, V and C touch memory: 107 us, and no
// row length, odd ones included, leaves the tensor cores (3 sequences of 197 tokens: 750 -> 87 us a layer).
//
// What bounds it: the integer arithmetic of the softmax, about 20 instructions per score (two RESCALEs, a table
// look-up with interpolation, a 64-bit product); the two products take under a tenth of that.  Hence
//   * both RESCALEs from 32-bit words (scaleHigh32); the first one's operand is never positive and the second one's never
//     negative, so their double-rounding terms are constants;
//   * a table entry holds (value, step to the next value) as two int16, so that one look-up and one two-way dot product
//     give value * 128 + step * fraction;
//   * P is stored minus its zero point, as unsigned bytes, so that the second product needs no correction row;
//   * packing saturates (cvt.pack.sat), which is the clamp of the last RESCALE.
// Sixteen warps share the 128 x keys scores (four per quarter of the tensor-memory lanes, 16-column slices in turn) and
// exchange row maxima and row sums through shared memory.  Up to 192 keys a block has eight warps, so that two blocks
// fit an SM and one's products run under the other's softmax.  The next tile's Q and K are fetched as soon as the score
// product is done with them, V after the context product.
#include <algorithm>

#include "attention_i8.hpp"
#include "tcgen05_common.cuh"

namespace mlel {

namespace {

using namespace tc;

constexpr int kRowBytes = 128; // a SWIZZLE_128B row: one query or key, up to 128 bytes of head dimension

struct AttentionParams {
    const int8_t *q, *k, *v;
    int8_t *out;
    int32_t Sq, Sk, d, keysPad; // keysPad: keys rounded up to the 32 of an MMA's K step
    uint32_t tiles;
    FastDiv queryTiles, heads;
    int64_t qStride[3], kStride[3], vStride[3], oStride[3]; // bytes: sequence batch, head, token
    const int16_t *expTable, *recipTable;
    AttentionPlan plan;
};

struct AttentionShared {
    uint64_t scoresDone, contextDone;
    uint32_t tmemBase;
    int32_t failed;
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
__device__ __forceinline__ void tmemStore16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
                 "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
                 "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                 "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}

// Rows of `d` bytes into SWIZZLE_128B rows (16-byte piece j of row r at piece j ^ (r & 7)), as asynchronous copies;
// rows past `rows` and pieces past d (up to the 32 bytes of an MMA's K step) are zero-filled.
__device__ __forceinline__ void loadRows(uint8_t *dst, const int8_t *src, int64_t stride, int rows, int rowsPad, int d,
                                         int threads) {
    const int pieces = (d + 31) / 32 * 2;
    const uint32_t base = smemAddr(dst);
    for (int i = threadIdx.x; i < rowsPad * pieces; i += threads) {
        const int r = i / pieces, j = i - r * pieces;
        const bool live = r < rows && 16 * j < d;
        const int8_t *from = live ? src + int64_t(r) * stride + 16 * j : src;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(base + uint32_t(r * kRowBytes + ((j ^ (r & 7)) << 4))),
                     "l"(from), "r"(live ? 16u : 0u)
                     : "memory");
    }
}

template <int WARPS, bool UNSIGNED_P>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 8 ? 2 : 1) attentionI8Kernel(const __grid_constant__ AttentionParams p) {
    constexpr int kThreads = WARPS * 32;
    constexpr int kGroups = WARPS / 4; // warps per quarter of the tensor-memory lanes
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
    uint32_t columns = 32;
    while (columns < uint32_t(p.keysPad) || columns < uint32_t(p.d)) {
        columns *= 2;
    }

    if (threadIdx.x == 0) {
        mbarInit(&shared->scoresDone, 1);
        mbarInit(&shared->contextDone, 1);
        shared->failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = threadIdx.x; i < 512; i += kThreads) {
        const int32_t value = p.expTable[i], next = p.expTable[i + 1];
        expLut[i] = (uint32_t(value) << 16) | (uint32_t(next - value) & 0xffffu); // the step fits int16 (fuseAttention)
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(&shared->tmemBase)),
                     "r"(columns)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmemBase = shared->tmemBase;
    gridDependencySync(); // from here on activations are read and written

    struct Tile {
        uint32_t n, h;
        int q0;
    };
    const auto tileOf = [&](uint32_t t) {
        const uint32_t b = fastDiv(t, p.queryTiles), n = fastDiv(b, p.heads);
        return Tile{n, b - n * p.heads.d, int(t - b * p.queryTiles.d) * BM};
    };
    const auto loadQK = [&](const Tile &t) {
        loadRows(tileQ, p.q + t.n * p.qStride[0] + t.h * p.qStride[1] + t.q0 * p.qStride[2], p.qStride[2], p.Sq - t.q0, BM, p.d,
                 kThreads);
        loadRows(tileK, p.k + t.n * p.kStride[0] + t.h * p.kStride[1], p.kStride[2], p.Sk, p.keysPad, p.d, kThreads);
    };
    const auto loadV = [&](const Tile &t) {
        loadRows(tileV, p.v + t.n * p.vStride[0] + t.h * p.vStride[1], p.vStride[2], p.Sk, p.keysPad, p.d, kThreads);
    };
    const auto commitCopies = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
    const auto waitAllButLastCopies = [] {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // the tensor core reads what the copies wrote
    };
    // the warps of one quarter, i.e. of the same 32 rows
    const auto quarterSync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(1 + quarter), "n"(kGroups * 32) : "memory"); };

    const AttentionPlan &a = p.plan;
    const int slices = p.keysPad / 16;
    const uint32_t laneAddr = tmemBase + (uint32_t(quarter * 32) << 16);
    uint32_t parity = 0;

    uint32_t t = blockIdx.x;
    if (t < p.tiles) {
        const Tile first = tileOf(t);
        loadQK(first);
        commitCopies();
        loadV(first);
        commitCopies();
    }
    for (; t < p.tiles; t += gridDim.x, parity ^= 1u) {
        const Tile tile = tileOf(t);
        const bool more = t + gridDim.x < p.tiles;
        waitAllButLastCopies(); // Q and K; V may still be under way
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        if (shared->failed != 0) {
            break;
        }
        if (threadIdx.x == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t descQ = smemDesc(smemAddr(tileQ), 16, 1024), descK = smemDesc(smemAddr(tileK), 16, 1024);
            for (int n0 = 0; n0 < p.keysPad; n0 += 256) {
                const int n = min(256, p.keysPad - n0);
                for (int ks = 0; ks * UMMA_K < p.d; ++ks) {
                    umma(tmemBase + uint32_t(n0), descQ + uint64_t(2 * ks), descK + uint64_t(n0 * (kRowBytes >> 4) + 2 * ks),
                         instrDesc(n, false), ks > 0 ? 1u : 0u);
                }
            }
            ummaCommit(&shared->scoresDone);
        }
        if (!mbarWait(&shared->scoresDone, parity, 71)) {
            shared->failed = 1;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (more) {
            loadQK(tileOf(t + gridDim.x));
        }
        commitCopies();

        // ---- row maximum
        int32_t top = int32_t(0x80000000u);
        for (int c = columnGroup; c < slices; c += kGroups) {
            uint32_t s[16];
            tmemLoad16(laneAddr + uint32_t(16 * c), s);
            tmemWait16(s);
            const int live = p.Sk - 16 * c; // columns of real keys in this slice
            if (live >= 16) {
#pragma unroll
                for (int j = 0; j < 16; j += 2) {
                    top = __vimax3_s32(top, int32_t(s[j]), int32_t(s[j + 1]));
                }
            } else {
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    top = j < live ? max(top, int32_t(s[j])) : top;
                }
            }
        }
        partMax[columnGroup * BM + row] = top;
        quarterSync();
#pragma unroll
        for (int g = 0; g < kGroups; ++g) {
            top = max(top, partMax[g * BM + row]);
        }

        // ---- exponentials, in place; row sum
        const int32_t top4 = int32_t(uint32_t(top) * 4u);
        uint32_t sum = 0;
        for (int c = columnGroup; c < slices; c += kGroups) {
            uint32_t s[16];
            tmemLoad16(laneAddr + uint32_t(16 * c), s);
            tmemWait16(s);
            const int live = p.Sk - 16 * c;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const int32_t x4 = int32_t(s[j] * 4u) - top4;
                const int32_t scaled = scaleHigh32<false>(x4, a.diffMult, a.diffRound) >> a.diffShift;
                const uint32_t u = uint32_t(min(__viaddmax_s32(scaled, a.diffAdd, a.diffLo), a.diffHi)); // int16 + 32768
                const uint32_t entry = *reinterpret_cast<const uint32_t *>(reinterpret_cast<const uint8_t *>(expLut) + ((u >> 5) & ~3u));
                s[j] = uint32_t(dp2aLow(entry, (u & 0x7fu) | 0x8000u, 0));
            }
            if (live >= 16) {
#pragma unroll
                for (int j = 0; j < 16; j += 2) {
                    sum += s[j] + s[j + 1];
                }
            } else {
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    s[j] = j < live ? s[j] : 0u;
                    sum += s[j];
                }
            }
            tmemStore16(laneAddr + uint32_t(16 * c), s);
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
        for (int c = columnGroup; c < slices; c += kGroups) {
            uint32_t s[16];
            tmemLoad16(laneAddr + uint32_t(16 * c), s);
            tmemWait16(s);
            uint32_t packed[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                int32_t y[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint64_t prod = uint64_t(int64_t(int32_t(s[4 * q + j])) * int64_t(recip)) + uint64_t(a.mulRound);
                    const uint32_t x = __funnelshift_r(uint32_t(prod), uint32_t(prod >> 32), uint32_t(a.mulShift));
                    y[j] = scaleHigh32<false>(int32_t(x * 4u), a.probMult, a.probRound) >> a.probShift;
                }
                packed[q] = packSat<UNSIGNED_P>(y[1], y[0], packSat<UNSIGNED_P>(y[3], y[2], 0u));
            }
            // 16-byte piece c & 7 of this row in the 128-key block c >> 3
            *reinterpret_cast<uint4 *>(tileP + (c >> 3) * (BM * BK) + row * BK + (((c & 7) ^ (row & 7)) << 4)) =
                make_uint4(packed[0], packed[1], packed[2], packed[3]);
        }
        waitAllButLastCopies(); // V; the next tile's Q and K may still be under way.  The fence also covers P
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        if (threadIdx.x == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // the context takes the first d columns: every score has been read
            const uint32_t idesc = instrDesc(p.d, true) & (UNSIGNED_P ? ~(7u << 7) : ~0u); // A format 0: unsigned 8-bit
            const uint64_t descP = smemDesc(smemAddr(tileP), 16, 1024), descV = smemDesc(smemAddr(tileV), BK * 128, 1024);
            for (int ks = 0; ks * UMMA_K < p.keysPad; ++ks) {
                umma(tmemBase, descP + uint64_t((ks >> 2) * ((BM * BK) >> 4) + 2 * (ks & 3)),
                     descV + uint64_t(ks * ((UMMA_K * kRowBytes) >> 4)), idesc, ks > 0 ? 1u : 0u);
            }
            ummaCommit(&shared->contextDone);
        }
        if (!mbarWait(&shared->contextDone, parity, 72)) {
            shared->failed = 1;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (more) {
            loadV(tileOf(t + gridDim.x));
        }
        commitCopies();

        // ---- context rows
        int8_t *dst = p.out + tile.n * p.oStride[0] + tile.h * p.oStride[1] + int64_t(tile.q0 + row) * p.oStride[2];
        for (int c = columnGroup; 16 * c < p.d; c += kGroups) {
            uint32_t s[16];
            tmemLoad16(laneAddr + uint32_t(16 * c), s);
            tmemWait16(s);
            uint32_t packed[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                uint32_t w = 0;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    w |= uint32_t(uint8_t(fastRescale(a.context, int32_t(s[4 * q + j]), a.contextOutZp, a.contextLo, a.contextHi)))
                         << (8 * j);
                }
                packed[q] = w;
            }
            if (tile.q0 + row < p.Sq) {
                *reinterpret_cast<uint4 *>(dst + 16 * c) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmemBase), "r"(columns) : "memory");
    }
}

size_t attentionSmem(int keysPad, int warps) {
    return 1024 + size_t(BM) * kRowBytes + 2 * size_t(keysPad) * kRowBytes + size_t((keysPad + 127) / 128) * BM * BK + 512 * 4 +
           2 * size_t(warps / 4) * BM * 4 + sizeof(AttentionShared);
}

template <int WARPS>
int launchAttention(const AttentionParams &p, bool unsignedP, cudaStream_t s) {
    const size_t smem = attentionSmem(p.keysPad, WARPS);
    auto kernel = unsignedP ? attentionI8Kernel<WARPS, true> : attentionI8Kernel<WARPS, false>;
    if (!allowDynamicSmem(reinterpret_cast<const void *>(kernel), attentionSmem(WARPS == 8 ? kAttentionTwoBlockKeys : kAttentionMaxKeys, WARPS))) {
        return MLEL_ERROR_DEVICE;
    }
    const int grid = int(std::min<int64_t>(p.tiles, int64_t(smCount()) * (WARPS == 8 ? 2 : 1)));
    if (launchDependent(kernel, grid, WARPS * 32, smem, s, p) != cudaSuccess) {
        setLastError(std::string("attention: ") + cudaGetErrorString(cudaGetLastError()));
        return MLEL_ERROR_DEVICE;
    }
    return MLEL_SUCCESS;
}

} // namespace

int attentionErrorWord() { return readErrorWord(); }

int attentionFused(const AttentionPlan &plan, const TView &q, const TView &k, const TView &v, const TView &expTable,
                   const TView &recipTable, const TView &out, cudaStream_t s) {
    AttentionParams p{};
    p.plan = plan;
    p.q = reinterpret_cast<const int8_t *>(q.ptr);
    p.k = reinterpret_cast<const int8_t *>(k.ptr);
    p.v = reinterpret_cast<const int8_t *>(v.ptr);
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
        p.qStride[i] = plan.qStride[i], p.kStride[i] = plan.kStride[i];
        p.vStride[i] = plan.vStride[i], p.oStride[i] = plan.oStride[i];
    }
    if (((reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.k) | reinterpret_cast<uintptr_t>(p.v) |
          reinterpret_cast<uintptr_t>(p.out)) & 15u) != 0) {
        setLastError("attention: operands must be 16-byte aligned");
        return MLEL_ERROR_UNKNOWN;
    }
    return p.keysPad <= kAttentionTwoBlockKeys ? launchAttention<8>(p, plan.unsignedProb, s)
                                              : launchAttention<16>(p, plan.unsignedProb, s);
}

} // namespace mlel
