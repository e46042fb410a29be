// int8 convolution / matrix product for problems that would leave most of the GPU idle: one image's layers, a
// classifier's product, the late stages of a small batch.
//
//   D[oc, pix] = sum_k W[oc, k] * X[pix, k]      one tile = 128 output channels x BNP (32 or 64) pixels,
//                                                its K blocks shared by a cluster of SPLIT CTAs
//
// What bounds these problems is latency, not work.  A ResNet-50-shaped dispatch of one image spent 7.2 us a layer in the
// channel-major kernel (clock stamps of CTA 0): 0.31 us per K block, one after the other -- 5.3 us for a 3x3 layer with
// 256 channels, on 4 SMs --, 1.0-2.2 us in the epilogue of a 128 x 128 tile, and 2.4-3.1 us from there to the next layer's
// first operand.  Here
//   * tiles are narrow, so that many SMs share the epilogue and the pixel loads, and the K blocks of a tile are split
//     over up to eight CTAs of a cluster.  Every CTA finishes BNP / SPLIT pixels: the others send it their int32 partial
//     sums with st.async, which completes on its mbarrier, so that no cluster-wide barrier lies behind the products
//     (with partial sums in the senders' shared memory and two cluster barriers this part took 1.7 us of a layer's 5).
//     Integer sums wrap, so the order does not change the result;
//   * sixteen epilogue warps: a thread has BNP / SPLIT / 4 results (a residual tail is three RESCALEs more, and 32 results
//     a thread took 3.5 us);
//   * weights and the epilogue's constants do not depend on the launch before (unless it made them: a product of two
//     activations): they are fetched ahead of griddepcontrol.wait, and a CTA is small enough (about 100 KB, 32 or 64 columns of tensor memory) to be resident
//     beside the CTAs of the launches around it;
//   * results go from registers to memory: 32 lanes hold 32 neighbouring channels of a pixel.
// The arithmetic is the other kernels' (fastRescale); a residual tail is looked up in its table where there is one.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "gemm_i8_tcgen05.hpp"
#include "tcgen05_common.cuh"

namespace mlel {
namespace {

using namespace tc;

constexpr int kSmallChannels = 128; // UMMA M
constexpr int kSmallEpilogueWarps = 16, kSmallTmaWarp = 16, kSmallMmaWarp = 17, kSmallThreads = 576;
constexpr int smallStages(int bnp) { return bnp == 32 ? 4 : 3; } // with the partial sums 96 and 104 KB: two CTAs fit an SM

struct __align__(8) SmallBarriers {
    uint64_t full[4], empty[4];
    uint64_t accFull, sumsFull;
    uint32_t tmemBase, pad;
};

__device__ __forceinline__ void clusterArrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void clusterWait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t clusterAddr(uint32_t localAddr, uint32_t rank) {
    uint32_t addr;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(localAddr), "r"(rank));
    return addr;
}
// 16 bytes to a CTA of the cluster, counted by that CTA's mbarrier
__device__ __forceinline__ void sendFour(uint32_t addr, uint32_t bar, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%2, %3, %4, %5}, [%1];" ::"r"(addr), "r"(bar),
                 "r"(a), "r"(b), "r"(c), "r"(d)
                 : "memory");
}
__device__ __forceinline__ void prefetchMap(const CUtensorMap *map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// A residual tail: looked up in its table, or (where it has none) evaluated.
enum : int { kNoTail = 0, kTailTable = 1, kTailArithmetic = 2 };

// IM2COL: mapX is an im2col map of the NHWC input and mapW a {IC, taps, OC} map; else mapX is a plain pixel matrix.
template <int BNP, int SPLIT, bool IM2COL, int TAIL, bool TABLE = false>
__global__ void __launch_bounds__(kSmallThreads, 2)
gemmI8Small(const __grid_constant__ CUtensorMap mapX, const __grid_constant__ CUtensorMap mapW, const __grid_constant__ GemmI8Params p) {
    constexpr bool RESIDUAL = TAIL != kNoTail;
    constexpr int kStages = smallStages(BNP);
    constexpr int kTileW = kSmallChannels * BK, kTileX = BNP * BK;
    constexpr int kPixels = BNP / SPLIT; // pixels that this CTA finishes
    constexpr int kMine = kPixels / 4;   // and this thread
    extern __shared__ uint8_t rawSmem[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(rawSmem) + 1023) & ~uintptr_t(1023));
    uint8_t *tilesW = smem, *tilesX = smem + kStages * kTileW;
    // partial sums of this CTA's pixels: [sender][groups of four pixels][128 channels][4 pixels]
    uint8_t *sums = smem + kStages * (kTileW + kTileX);
    SmallBarriers *bars = reinterpret_cast<SmallBarriers *>(sums + (SPLIT > 1 ? BNP * kSmallChannels * 4 : 0));

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = int(blockIdx.x) % SPLIT;
    const uint32_t tile = blockIdx.x / SPLIT;
    // pixel tile fastest: neighbouring clusters read the same weights
    const uint32_t cTile = fastDiv(tile, p.divTiles0), pTile = tile - cTile * p.divTiles0.d;
    const int c0 = int(cTile) * kSmallChannels, m0 = int(pTile) * BNP;
    const int numKb = IM2COL ? p.KH * p.KW * p.kbPerTap : (p.K + BK - 1) / BK;
    const int kb0 = numKb * rank / SPLIT, kbCount = numKb * (rank + 1) / SPLIT - kb0;

    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (threadIdx.x == kSmallTmaWarp * 32) {
        prefetchMap(&mapW);
        prefetchMap(&mapX);
        for (int s = 0; s < kStages; ++s) {
            mbarInit(&bars->full[s], 1);
            mbarInit(&bars->empty[s], 1);
        }
        mbarInit(&bars->accFull, 1);
        mbarInit(&bars->sumsFull, 1);
        if (SPLIT > 1) {
            mbarArriveExpectTx(&bars->sumsFull, uint32_t(BNP * kSmallChannels * 4));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kSmallMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(&bars->tmemBase)),
                     "r"(uint32_t(BNP))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmemBase = bars->tmemBase;
    if (SPLIT > 1) {
        clusterArrive(); // waited for before the first partial sum is sent: every CTA's barriers are ready
    }

    // Epilogue warps: a channel per thread (its lane of tensor memory), a quarter of this CTA's pixels per four warps
    const int group = warp >> 2;
    const int oc = c0 + (warp & 3) * 32 + lane;
    const bool ocValid = oc < p.N;
    const int firstPixel = m0 + rank * kPixels + group * kMine;
    FastRescale main{};
    int32_t corr[kMine];

    if (warp == kSmallTmaWarp) {
        if (lane == 0) {
            // (running positions on the K axis: the divisions that they take are done once)
            const int tap0 = IM2COL ? kb0 / p.kbPerTap : 0, cb0 = IM2COL ? (kb0 - tap0 * p.kbPerTap) * BK : kb0 * BK;
            int tapW = tap0, cbW = cb0, stageW = 0;
            const auto loadW = [&] {
                uint64_t *full = &bars->full[stageW];
                mbarArriveExpectTx(full, uint32_t(kTileW + kTileX));
                if (IM2COL) {
                    tmaLoad3d(&mapW, tilesW + stageW * kTileW, full, cbW, tapW, c0);
                } else {
                    tmaLoad3d(&mapW, tilesW + stageW * kTileW, full, cbW, c0, 0);
                }
                cbW += BK;
                if (IM2COL && cbW >= p.IC) {
                    cbW = 0;
                    ++tapW;
                }
                stageW = stageW + 1 == kStages ? 0 : stageW + 1;
            };
            int w0 = 0, h0 = 0, n0 = 0; // first tap of the tile's first window
            int cbX = cb0, stageX = 0, ky = IM2COL ? tap0 / p.KW : 0, kx = tap0 - ky * p.KW;
            if (IM2COL) {
                n0 = int(fastDiv(uint32_t(m0), p.divPlane));
                const int rem = m0 - n0 * p.OH * p.OW, oy = int(fastDiv(uint32_t(rem), p.divOW));
                h0 = oy * p.strideY - p.padTop, w0 = (rem - oy * p.OW) * p.strideX - p.padLeft;
            }
            const auto loadX = [&] {
                uint64_t *full = &bars->full[stageX];
                if (IM2COL) {
                    tmaLoadIm2col4d(&mapX, tilesX + stageX * kTileX, full, cbX, w0, h0, n0, uint16_t(kx * p.dilX),
                                    uint16_t(ky * p.dilY));
                } else {
                    tmaLoad3d(&mapX, tilesX + stageX * kTileX, full, cbX, m0, 0);
                }
                cbX += BK;
                if (IM2COL && cbX >= p.IC) {
                    cbX = 0;
                    if (++kx == p.KW) {
                        kx = 0;
                        ++ky;
                    }
                }
                stageX = stageX + 1 == kStages ? 0 : stageX + 1;
            };
            const int ahead = min(kbCount, kStages);
            if (p.lateOperand != 0) {
                asm volatile("griddepcontrol.wait;" ::: "memory");
            }
            for (int i = 0; i < ahead; ++i) {
                loadW();
            }
            asm volatile("griddepcontrol.wait;" ::: "memory"); // the pixels are the launch before's results
            for (int i = 0; i < ahead; ++i) {
                loadX();
            }
            for (int i = ahead; i < kbCount; ++i) {
                if (!mbarWait(&bars->empty[i % kStages], uint32_t(i / kStages - 1) & 1u, 81)) {
                    break;
                }
                loadW();
                loadX();
            }
        }
        __syncwarp();
    } else if (warp == kSmallMmaWarp) {
        // The whole warp (see ummaBlockPeek).  From one divergent lane a K block took 0.3-0.4 us between its operands' arrival and
        // the next one's MMAs: 1.1 us of a layer's 4 with three K blocks, 2.3 with six.  (All K blocks on one barrier, one wait and
        // one train of MMAs: slower, one image 228 us against 219 -- the first block's MMAs run while the others arrive.)  A wait
        // that runs out only ends the waiting, the recorded error tells.
        const DescWords descW = descWords(smemDesc(smemAddr(tilesW), 16, 1024)), descX = descWords(smemDesc(smemAddr(tilesX), 16, 1024));
        int left = IM2COL ? p.IC - kb0 % p.kbPerTap * BK : p.K - kb0 * BK; // bytes of K from here to the end of the tap or row
        bool failed = false;
        uint32_t ready = 0, phase = 0;
        int s = 0;
        for (int i = 0; i < kbCount; ++i) {
            if (ready == 0) {
                failed = failed || !mbarWait(&bars->full[s], phase, 82);
            }
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int sNext = s + 1 == kStages ? 0 : s + 1;
            const uint32_t phaseNext = sNext == 0 ? phase ^ 1u : phase;
            ready = ummaBlockPeek(tmemBase, {descW.low + uint32_t(s * (kTileW >> 4)), descW.high}, 2,
                                  {descX.low + uint32_t(s * (kTileX >> 4)), descX.high}, 2, instrDesc(BNP, false), i > 0 ? 1u : 0u,
                                  ummaCountFor(left), &bars->empty[s], &bars->full[sNext], phaseNext);
            left = IM2COL && left <= BK ? p.IC : left - BK;
            s = sNext;
            phase = phaseNext;
        }
        ummaCommit(&bars->accFull);
        __syncwarp();
    } else {
        const int ci = p.epi.main.perChannel && ocValid ? oc : 0;
        main = makeFastRescale(__ldg(p.epi.main.mult + ci), int32_t(__ldg(p.epi.main.shift + ci)), p.epi.main.inZp,
                               p.epi.main.doubleRound != 0);
        if (p.lateOperand != 0) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
        }
#pragma unroll
        for (int j = 0; j < kMine; ++j) {
            int cls = p.baseClass;
            if (p.rowClass != nullptr && firstPixel + j < p.M) {
                const uint32_t m = uint32_t(firstPixel + j), rem = m - fastDiv(m, p.divPlane) * p.divPlane.d;
                const uint32_t oy = fastDiv(rem, p.divOW);
                cls = int(__ldg(p.rowClass + oy)) * p.numColClasses + int(__ldg(p.colClass + (rem - oy * uint32_t(p.OW))));
            }
            corr[j] = ocValid ? p.corr[int64_t(cls) * p.N + oc] : 0;
        }
        asm volatile("griddepcontrol.wait;" ::: "memory"); // from here on activations are read and written
    }

    if (SPLIT > 1) {
        clusterWait();
    }
    if (warp < kSmallEpilogueWarps) {
        uint32_t acc[kMine];
        int8_t shortcut[kMine];
        if (RESIDUAL) {
            const int8_t *row = p.epi.shortcut + int64_t(firstPixel) * p.ldOut + oc;
#pragma unroll
            for (int j = 0; j < kMine; ++j) {
                shortcut[j] = ocValid && firstPixel + j < p.M ? row[int64_t(j) * p.ldOut] : int8_t(0);
            }
        }
        mbarWait(&bars->accFull, 0, 83);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // columns (pixels of the tile) of this warp: a quarter of them
        constexpr int kColumns = BNP / 4;
        const uint32_t taddr = tmemBase + (uint32_t((warp & 3) * 32) << 16) + uint32_t(group * kColumns);
        uint32_t r[16];
        if (kColumns == 8) {
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                         : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                         : "r"(taddr)
                         : "memory");
#pragma unroll
            for (int j = 8; j < 16; ++j) {
                r[j] = 0;
            }
        } else {
            tmemLoad16(taddr, r);
        }
        tmemWait16(r);
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        if (SPLIT == 1) {
#pragma unroll
            for (int j = 0; j < kMine; ++j) {
                acc[j] = r[j];
            }
        } else {
            const uint32_t base = smemAddr(sums), bar = smemAddr(&bars->sumsFull);
            const uint32_t channel = uint32_t((warp & 3) * 32 + lane);
#pragma unroll
            for (int q = 0; q < kColumns / 4; ++q) {
                const int pixel = group * kColumns + 4 * q, owner = pixel / kPixels, four = (pixel - owner * kPixels) / 4;
                const uint32_t slot = uint32_t((rank * (kPixels / 4) + four) * kSmallChannels) + channel;
                sendFour(clusterAddr(base + slot * 16u, uint32_t(owner)), clusterAddr(bar, uint32_t(owner)), r[4 * q], r[4 * q + 1],
                         r[4 * q + 2], r[4 * q + 3]);
            }
            // (longer than the senders' own waits: a sender that gave up still sends before this CTA may leave)
            mbarWaitLimit(&bars->sumsFull, 0, 84, 3 * kWaitLimitCycles);
#pragma unroll
            for (int j = 0; j < kMine; ++j) {
                const int pixel = group * kMine + j;
                acc[j] = 0;
#pragma unroll
                for (int sender = 0; sender < SPLIT; ++sender) {
                    const uint32_t slot = uint32_t((sender * (kPixels / 4) + (pixel >> 2)) * kSmallChannels) + channel;
                    uint32_t v;
                    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(base + slot * 16u + uint32_t(pixel & 3) * 4u) : "memory");
                    acc[j] += v;
                }
            }
        }
        FastRescale fa{}, fb{}, fo{};
        if (TAIL == kTailArithmetic) {
            fa = makeFastRescale(__ldg(p.epi.a.mult), int32_t(__ldg(p.epi.a.shift)), p.epi.a.inZp, p.epi.a.doubleRound != 0);
            fb = makeFastRescale(__ldg(p.epi.b.mult), int32_t(__ldg(p.epi.b.shift)), p.epi.b.inZp, p.epi.b.doubleRound != 0);
            fo = makeFastRescale(__ldg(p.epi.out.mult), int32_t(__ldg(p.epi.out.shift)), p.epi.out.inZp, p.epi.out.doubleRound != 0);
        }
        int8_t *dst = p.out8 + int64_t(firstPixel) * p.ldOut + oc;
#pragma unroll
        for (int j = 0; j < kMine; ++j) {
            int32_t v = fastRescale(main, int32_t(acc[j] + uint32_t(corr[j])), p.epi.main.outZp, p.epi.main.lo, p.epi.main.hi);
            if (TAIL == kTailTable) {
                // The whole tail is a byte of this table, a load from cache where the three RESCALEs took 0.8 us of a layer's 4
                // (one image of the ResNet-50 shape 222.1 -> 219.4 us, 32 of the MobileNetV2 shape 481 -> 473.5).
                v = int32_t(__ldg(p.residualTable + (v + 128) * GemmI8Params::kResidualRowBytes + int32_t(uint8_t(shortcut[j]))));
            } else if (TAIL == kTailArithmetic) {
                const int32_t ta = fastRescale(fa, v, p.epi.a.outZp, p.epi.a.lo, p.epi.a.hi);
                const int32_t tb = fastRescale(fb, int32_t(shortcut[j]), p.epi.b.outZp, p.epi.b.lo, p.epi.b.hi);
                v = fastRescale(fo, int32_t(uint32_t(ta) + uint32_t(tb)), p.epi.out.outZp, p.epi.out.lo, p.epi.out.hi);
            }
            if (TABLE) {
                v = int32_t(__ldg(p.epi.table + 128 + v));
            }
            if (ocValid && firstPixel + j < p.M) {
                dst[int64_t(j) * p.ldOut] = int8_t(v);
            }
        }
    }
    __syncthreads();
    if (warp == kSmallMmaWarp) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmemBase), "r"(uint32_t(BNP)) : "memory");
    }
}

template <int BNP, int SPLIT, bool IM2COL, int TAIL, bool TABLE = false>
int launchSmall(const CUtensorMap &mapX, const CUtensorMap &mapW, const GemmI8Params &p, int tiles, cudaStream_t s) {
    constexpr size_t smem = size_t(smallStages(BNP)) * (kSmallChannels + BNP) * BK +
                            (SPLIT > 1 ? size_t(BNP) * kSmallChannels * 4 : 0) + sizeof(SmallBarriers) + 1024;
    auto kernel = gemmI8Small<BNP, SPLIT, IM2COL, TAIL, TABLE>;
    if (!allowDynamicSmem(reinterpret_cast<const void *>(kernel), smem)) {
        return MLEL_ERROR_DEVICE;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(unsigned(tiles * SPLIT));
    cfg.blockDim = dim3(kSmallThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attrs[2]{};
    attrs[0].id = cudaLaunchAttributeClusterDimension;
    attrs[0].val.clusterDim.x = SPLIT, attrs[0].val.clusterDim.y = attrs[0].val.clusterDim.z = 1;
    attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attrs;
    cfg.numAttrs = dependentLaunches() ? 2 : 1;
    const cudaError_t err = cudaLaunchKernelEx(&cfg, kernel, mapX, mapW, p);
    if (err != cudaSuccess) {
        setLastError(std::string("small int8 GEMM launch: ") + cudaGetErrorString(err));
        return MLEL_ERROR_DEVICE;
    }
    return MLEL_SUCCESS;
}

template <int BNP, int SPLIT>
int launchSmallMode(const CUtensorMap &mapX, const CUtensorMap &mapW, const GemmI8Params &p, int tiles, bool im2col, cudaStream_t s) {
    const int tail = !p.epi.hasResidual ? kNoTail : (p.residualTable != nullptr ? kTailTable : kTailArithmetic);
    if (im2col) {
        return tail == kNoTail      ? launchSmall<BNP, SPLIT, true, kNoTail>(mapX, mapW, p, tiles, s)
               : tail == kTailTable ? launchSmall<BNP, SPLIT, true, kTailTable>(mapX, mapW, p, tiles, s)
                                    : launchSmall<BNP, SPLIT, true, kTailArithmetic>(mapX, mapW, p, tiles, s);
    }
    if (p.epi.table != nullptr) {
        return launchSmall<BNP, SPLIT, false, kNoTail, true>(mapX, mapW, p, tiles, s);
    }
    return tail == kNoTail      ? launchSmall<BNP, SPLIT, false, kNoTail>(mapX, mapW, p, tiles, s)
           : tail == kTailTable ? launchSmall<BNP, SPLIT, false, kTailTable>(mapX, mapW, p, tiles, s)
                                : launchSmall<BNP, SPLIT, false, kTailArithmetic>(mapX, mapW, p, tiles, s);
}

template <int BNP>
int launchSmallSplit(const CUtensorMap &mapX, const CUtensorMap &mapW, const GemmI8Params &p, int tiles, int split, bool im2col,
                     cudaStream_t s) {
    switch (split) {
    case 1:
        return launchSmallMode<BNP, 1>(mapX, mapW, p, tiles, im2col, s);
    case 2:
        return launchSmallMode<BNP, 2>(mapX, mapW, p, tiles, im2col, s);
    case 4:
        return launchSmallMode<BNP, 4>(mapX, mapW, p, tiles, im2col, s);
    default:
        return launchSmallMode<BNP, 8>(mapX, mapW, p, tiles, im2col, s);
    }
}

} // namespace

bool smallKernelWants(int64_t pixels, int64_t channels, int halves) {
    const int64_t tiles = (pixels + 127) / 128 * ((channels + kSmallChannels - 1) / kSmallChannels);
    return tiles * halves <= 2 * smCount();
}

bool gemmI8SmallApplies(const GemmI8Problem &q, int *pixels, int *split) {
    const GemmI8Params &p = q.params;
    const int mode = tensorCoreTuning().smallKernel.load(std::memory_order_relaxed);
    if (mode == 0 || p.out8 == nullptr || !p.epi.hasMain || q.bMnMajor || q.batches != 1 || p.gatherTable != nullptr ||
        (q.aMatrix == nullptr && p.IC % 16 != 0)) {
        return false;
    }
    // Rule.  The other kernels' 128-pixel tiles would leave two thirds of the SMs without work; for some forms below, half of
    // them.  As many CTAs share a tile's K blocks as have two blocks each at
    // least, with at most two CTAs per SM -- neighbouring launches overlap, so a layer's own CTAs seldom meet (one image of the
    // ResNet-50-shaped graph: 248 us, at most one CTA per SM 267).  Tiles are 32 pixels wide.  With 64 a CTA of a larger split
    // has half the blocks but a larger share of the reduction: worth it only from some 13 blocks on that the narrow tile
    // would leave to a CTA (us a layer, narrow and wide: 2 x 33 x 33, 3x3, 160 <-> 128 channels, 4.5 blocks, 5.9 and 7.9; 14 x 14, 1x1,
    // 2048 <-> 1024, 4, 4.9 and 6.2; 19 x 19, 3x3, 768 -> 768, 13.5, 12.7 and 12.5; 4 x 33 x 33, 128 <-> 768, 27, 10.5 and 9.8; 2 x 56 x 56,
    // 2048 <-> 16, 144, 26.8 and 20.7).  While blocks took 0.3 us instead of 0.1 the wide one won wherever it allowed a larger split.
    const int sms = smCount();
    const int64_t cTiles = (p.N + kSmallChannels - 1) / kSmallChannels;
    const bool matrix = q.aMatrix != nullptr, product = p.OH == 0; // (a product has no image)
    // Beyond a third of the SMs, up to half for products of several blocks (of one block the gain is small: 3000 x 96 -> 384 4.4 and
    // 3.9, and the paired kernel keeps them) and two fifths for the others (240 shapes of 50 to 74 tiles of 128 x 128,
    // us a layer without and with): products of more than one channel tile and few blocks, which were the paired kernel's, 3201 x 256
    // -> 256 5.1 and 3.9, 867 x 1024 -> 320 5.0 and 4.3 (942 x 2048 -> 1000 8.6 and 9.5, not taken); 1x1 of two blocks at most, 59 x 37,
    // 160 -> 320 4.4 and 3.7 (102 x 17, 1024 -> 512 5.6 and 6.2, not taken; one channel tile, 36 x 93 x 2, 128 -> 128, 4.7 and 5.4); windows that
    // the window kernel does not read, 4 x 42 x 44, 3x3, 256 -> 96 9.0 and 7.9 (56 x 61, 16 -> 256 7.8 and 9.9).
    const bool further = matrix ? p.N > kSmallChannels && p.K <= (product ? 8 : 2) * BK : p.N > 64 && p.IC > 128;
    const int halves = !further ? kSmallKernelSurely : (product && p.K > BK ? 4 : 5);
    if (mode == 1 && !smallKernelWants(p.M, p.N, halves)) {
        return false;
    }
    const int numKb = q.aMatrix != nullptr ? (p.K + BK - 1) / BK : p.KH * p.KW * ((p.IC + 127) / 128);
    const auto splitFor = [&](int64_t tiles) {
        int s = 1;
        while (s < 8 && s * 4 <= numKb && tiles * s <= sms) {
            s *= 2;
        }
        return s;
    };
    const int split32 = splitFor(int64_t((p.M + 31) / 32) * cTiles), split64 = splitFor(int64_t((p.M + 63) / 64) * cTiles);
    const bool wide = split64 > split32 && numKb > 13 * split32;
    *pixels = wide ? 64 : 32;
    *split = wide ? split64 : split32;
    if (mode >= 100) { // an experiment's choice: pixels and split
        *pixels = mode / 100 == 1 ? 32 : 64;
        *split = std::min(mode % 100, numKb >= 8 ? 8 : (numKb >= 4 ? 4 : (numKb >= 2 ? 2 : 1)));
    }
    return true;
}

int gemmI8SmallLaunch(const GemmI8Problem &q, int pixels, int split, cudaStream_t s, bool *taken) {
    GemmI8Params p = q.params;
    p.batches = 1;
    p.progressOut = nullptr, p.progressIn = nullptr;
    if (p.epi.main.lo < -128 || p.epi.main.hi > 127) {
        p.residualTable = nullptr; // it is indexed by an int8 value
    }
    CUtensorMap mapX{}, mapW{};
    const bool im2col = q.aMatrix == nullptr;
    *taken = false;
    if (im2col) {
        if (!makeIm2colMap(&mapX, p.in, p.M / (p.OH * p.OW), p.H, p.W, p.IC, p.KH, p.KW, p.padTop, p.padLeft, p.OH, p.OW, p.strideY,
                           p.strideX, p.dilY, p.dilX, uint32_t(pixels)) ||
            !makeWeightTapMap(&mapW, q.bMatrix, p.IC, p.KH * p.KW, p.N, kSmallChannels)) {
            return MLEL_SUCCESS; // a geometry that the driver's im2col maps do not have: another kernel gathers
        }
        p.kbPerTap = (p.IC + 127) / 128;
    } else if (!makeMap(&mapX, q.aMatrix, uint64_t(p.K), uint64_t(p.M), 1, q.aRowBytes, q.aRowBytes * uint64_t(p.M), BK,
                        uint32_t(pixels)) ||
               !makeMap(&mapW, q.bMatrix, uint64_t(p.K), uint64_t(p.N), 1, q.bRowBytes, q.bRowBytes * uint64_t(p.N), BK,
                        kSmallChannels)) {
        return MLEL_ERROR_DEVICE;
    }
    *taken = true;
    g_tensorCoreLaunches[3].fetch_add(1, std::memory_order_relaxed);
    const int pixelTiles = (p.M + pixels - 1) / pixels, tiles = pixelTiles * ((p.N + kSmallChannels - 1) / kSmallChannels);
    p.divTiles0 = makeFastDiv(pixelTiles);
    p.divPlane = makeFastDiv(int64_t(p.OH) * p.OW), p.divOW = makeFastDiv(p.OW);
    return pixels == 32 ? launchSmallSplit<32>(mapX, mapW, p, tiles, split, im2col, s)
                        : launchSmallSplit<64>(mapX, mapW, p, tiles, split, im2col, s);
}

int smallErrorWord() { return readErrorWord(); }

} // namespace mlel
