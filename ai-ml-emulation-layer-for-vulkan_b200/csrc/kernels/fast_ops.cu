// Vectorised kernels for the packed int8 NHWC shapes that dominate real graphs.  Each has a generic
// counterpart in generic_ops.cu that defines the result; these only change how the bytes move.
#include <algorithm>

#include "device_common.cuh"
#include "gemm_i8_tcgen05.hpp"
#include "launch_overlapped.cuh"
#include "kernels.hpp"

namespace mlel {

namespace {

// ---- padded copy for convolutions whose channel count is not a multiple of 16 (an RGB stem) ---------
// Copies an NHWC int8 tensor [N][H][W][C] into [N][Hp][Wp][Cp] (Cp >= C a multiple of 4) at row offset
// padTop and column offset padLeft; the new channels and the border are zero.  One thread per 32-bit word
// of the copy: byte reads hit L1, writes are coalesced.
__global__ void padImageKernel(const int8_t *in, int8_t *out, int64_t words, int H, int W, int C,
                               int Hp, int Wp, int Cp, int padTop, int padLeft) {
    dependencySync();
    const int wordsPerPixel = Cp >> 2;
    for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < words; e += int64_t(gridDim.x) * blockDim.x) {
        int64_t pix = e / wordsPerPixel;
        const int c0 = int(e - pix * wordsPerPixel) * 4;
        const int x = int(pix % Wp) - padLeft;
        pix /= Wp;
        const int y = int(pix % Hp) - padTop;
        const int64_t n = pix / Hp;
        uint32_t word = 0;
        if (y >= 0 && y < H && x >= 0 && x < W) {
            const int8_t *src = in + ((n * H + y) * W + x) * C;
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                if (c0 + b < C) {
                    word |= uint32_t(uint8_t(src[c0 + b])) << (8 * b);
                }
            }
        }
        reinterpret_cast<uint32_t *>(out)[e] = word;
    }
}

// 16 bytes from any address, of which the first `valid` (1 to 16) exist; the others are zero.  Only aligned words that hold
// one of those bytes are read.
__device__ __forceinline__ int4 loadRagged16(const int8_t *p, int valid) {
    const uint32_t skip = uint32_t(reinterpret_cast<uintptr_t>(p)) & 3u;
    const uint32_t *words = reinterpret_cast<const uint32_t *>(p - skip);
    const int bytes = int(skip) + valid;
    uint32_t w[5], v[4];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        w[k] = 4 * k < bytes ? words[k] : 0u;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        v[k] = __funnelshift_r(w[k], w[k + 1], 8 * skip);
        const int left = valid - 4 * k;
        v[k] = left >= 4 ? v[k] : (left <= 0 ? 0u : v[k] & ((1u << (8 * left)) - 1u));
    }
    return make_int4(int(v[0]), int(v[1]), int(v[2]), int(v[3]));
}

// The same copy for channels padded to a multiple of 16: a thread makes 16 bytes of one pixel, from whole words.  BORDER:
// the copy has pixels that the image has not (false: rows of C bytes become rows of Cp).  Bound by its bytes.
template <bool BORDER>
__global__ void __launch_bounds__(256) padPixels16Kernel(const int8_t *in, int4 *out, uint32_t units, int H,
                                                         int W, int C, FastDiv perPixel, FastDiv divWp, FastDiv divHp, int padTop,
                                                         int padLeft) {
    dependencySync();
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < units; e += gridDim.x * blockDim.x) {
        const uint32_t pix = fastDiv(e, perPixel);
        const int c0 = int(e - pix * perPixel.d) * 16;
        int64_t from = pix;
        bool live = c0 < C;
        if (BORDER) {
            const uint32_t line = fastDiv(pix, divWp), n = fastDiv(line, divHp);
            const int x = int(pix - line * divWp.d) - padLeft, y = int(line - n * divHp.d) - padTop;
            live = live && unsigned(x) < unsigned(W) && unsigned(y) < unsigned(H);
            from = (int64_t(n) * H + y) * W + x;
        }
        out[e] = live ? loadRagged16(in + from * C + c0, min(16, C - c0)) : make_int4(0, 0, 0, 0);
    }
}

// ---- 16-byte units of four pixels for windows over at most four channels (gemm_i8_window.cu) --------------------
// Unit (y, x) of [N][Hu][Wu]: at stride 1 the pixels x - padLeft + 0..3 of row y, at stride 2 the pixels 2 x - padLeft + {0, 1}
// of the rows 2 y - padTop + {0, 1} (there padLeft and padTop are the paddings' remainders); four channels each, the
// missing ones and pixels outside the image zero.  Reads whole aligned words that hold a byte of the pixel.
template <int STRIDE>
__global__ void __launch_bounds__(256) gatherUnitsKernel(const int8_t *in, int4 *out, uint32_t units, int H,
                                                         int W, int C, FastDiv divWu, FastDiv divHu, int padTop, int padLeft) {
    dependencySync();
    const uint32_t mask = C == 4 ? 0xffffffffu : (1u << (8 * C)) - 1u;
    const uint32_t *words = reinterpret_cast<const uint32_t *>(in);
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < units; e += gridDim.x * blockDim.x) {
        const uint32_t line = fastDiv(e, divWu), n = fastDiv(line, divHu);
        const int x0 = int(e - line * divWu.d) * STRIDE - padLeft, y0 = int(line - n * divHu.d) * STRIDE - padTop;
        uint32_t px[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int x = x0 + (STRIDE == 1 ? k : k & 1), y = y0 + (STRIDE == 1 ? 0 : k >> 1);
            px[k] = 0;
            if (unsigned(x) < unsigned(W) && unsigned(y) < unsigned(H)) {
                const int64_t at = ((int64_t(n) * H + y) * W + x) * C;
                px[k] = __funnelshift_r(words[at >> 2], words[(at + C - 1) >> 2], 8 * (uint32_t(at) & 3u)) & mask;
            }
        }
        out[e] = make_int4(int(px[0]), int(px[1]), int(px[2]), int(px[3]));
    }
}

// The same copy for Cp == 4 and an even Wp (the RGB stem): one block per row of the copy, two pixels (one 8-byte
// store) per thread, no divisions in the element loop.
__global__ void __launch_bounds__(128) padImageRows4Kernel(const int8_t *in, int8_t *out, int H,
                                                          int W, int C, int Hp, int Wp, int padTop, int padLeft) {
    dependencySync();
    const int row = blockIdx.x; // n * Hp + yp
    const int n = row / Hp;
    const int y = row - n * Hp - padTop;
    const bool rowLive = y >= 0 && y < H;
    const int8_t *src = in + (int64_t(n) * H + (rowLive ? y : 0)) * W * C;
    uint2 *dst = reinterpret_cast<uint2 *>(out + int64_t(row) * Wp * 4);
    for (int q = threadIdx.x; 2 * q < Wp; q += blockDim.x) {
        uint32_t w[2] = {0u, 0u};
        if (rowLive) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int x = 2 * q + j - padLeft;
                if (x >= 0 && x < W) {
                    const int8_t *px = src + x * C;
                    for (int b = 0; b < C; ++b) {
                        w[j] |= uint32_t(uint8_t(px[b])) << (8 * b);
                    }
                }
            }
        }
        dst[q] = make_uint2(w[0], w[1]);
    }
}

// ---- transpose of MATMUL's second input [N][C][W] -> [N][W][Cp] with column sums ---------------------------
// Cp: C rounded up to a multiple of 16, the tail zero.  64 columns (w) of one batch belong to a cluster of `split` blocks
// that share the rows (c) and walk them in tiles of 64: 16-byte loads of the tile (the next tile's while this one is
// turned), byte transposition through shared memory, 16-byte stores; each thread keeps the running sum of the bytes it
// moved, four neighbouring lanes and then the cluster's blocks combine them into the column sum at the end.
// Latency bounds it where there are few columns: a tile is a chain of load, turn and store.
// ALIGNED: rows of B start on 16-byte boundaries.
template <bool ALIGNED>
__global__ void __launch_bounds__(256) transposeColsumKernel(const int8_t *b, int8_t *bt,
                                                             int32_t *corr, int C, int W, int Cp, int32_t za, int split) {
    dependencySync();
    __shared__ int8_t tile[64][64 + 16]; // [c][w], rows padded to spread the banks of the column reads
    __shared__ int32_t part[64];
    const int n = blockIdx.y;
    const int rank = int(blockIdx.x % unsigned(split)), w0 = int(blockIdx.x / unsigned(split)) * 64;
    const int t = threadIdx.x;
    const int8_t *src = b + int64_t(n) * C * W;
    int8_t *dst = bt + int64_t(n) * W * Cp;
    // load role: row (c) t / 4, 16-byte segment (w) t % 4; store role: column (w) t / 4, segment (c) t % 4
    const int lr = t >> 2, ls = (t & 3) * 16;
    int32_t sum = 0;
    const int tiles = (C + 63) / 64, first = tiles * rank / split * 64, last = tiles * (rank + 1) / split * 64;
    const auto fetch = [&](int c0) {
        if (c0 + lr >= C || w0 + ls >= W || c0 >= last) {
            return make_int4(0, 0, 0, 0);
        }
        const int8_t *p = src + int64_t(c0 + lr) * W + w0 + ls;
        return ALIGNED ? *reinterpret_cast<const int4 *>(p) : loadRagged16(p, min(16, W - (w0 + ls)));
    };
    int4 next = fetch(first);
    for (int c0 = first; c0 < last; c0 += 64) {
        *reinterpret_cast<int4 *>(&tile[lr][ls]) = next;
        next = fetch(c0 + 64);
        __syncthreads();
        uint32_t words[4] = {0, 0, 0, 0};
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int8_t x = tile[ls + i][lr];
            sum += x;
            words[i >> 2] |= uint32_t(uint8_t(x)) << (8 * (i & 3));
        }
        if (w0 + lr < W && c0 + ls < Cp) {
            *reinterpret_cast<int4 *>(dst + int64_t(w0 + lr) * Cp + c0 + ls) =
                make_int4(int(words[0]), int(words[1]), int(words[2]), int(words[3]));
        }
        __syncthreads();
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    if (split > 1) {
        if ((t & 3) == 0) {
            part[lr] = sum;
        }
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (rank == 0) {
            for (int r = 1; r < split; ++r) {
                uint32_t peer, v;
                const uint32_t local = uint32_t(__cvta_generic_to_shared(&part[lr]));
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(local), "r"(r));
                asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(peer));
                sum += int32_t(v);
            }
        }
        // block 0 has read the others' shared memory before they leave
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    if (rank == 0 && (t & 3) == 0 && w0 + lr < W) {
        corr[int64_t(n) * W + w0 + lr] = int32_t(uint32_t(0) - uint32_t(za) * uint32_t(sum));
    }
}

// ---- column sums of MATMUL's second input [N][C][W]: corr[n][w] = -za * sum_c b[n][c][w] --------------------
// For the tensor-core path that reads the operand where it lies (no transposed copy).  A block owns 64 columns
// of one batch: 4 lanes hold 16 columns each (one 16-byte load per row), 64 slices share the rows, eight rows in
// flight per thread.  Each byte goes through one dp4a against a one-hot selector, which sign-extends and accumulates it.
// A warp's eight slices join by shuffles, the eight warps in shared memory.
// The product is let in at once and waits for the sums only before its epilogue (kLateCorrections): 1024^3 14.5 -> 12.4 us.
__global__ void __launch_bounds__(256) columnSumKernel(const int8_t *b, int32_t *corr, int C, int W,
                                                       int32_t za) {
    __shared__ int32_t part[8][64];
    asm volatile("griddepcontrol.wait;" ::: "memory"); // first: the launch after this one relies on it
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int n = blockIdx.y;
    const int w0 = blockIdx.x * 64;
    const int seg = threadIdx.x & 3, slice = threadIdx.x >> 2;
    const int w = w0 + seg * 16;
    const int8_t *src = b + int64_t(n) * C * W + w;
    int32_t acc[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        acc[i] = 0;
    }
    if (w < W) { // W is a multiple of 16: a 16-byte segment is inside or outside as a whole
        for (int c0 = slice; c0 < C; c0 += 8 * 64) {
            int4 v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int c = c0 + 64 * u;
                v[u] = c < C ? *reinterpret_cast<const int4 *>(src + int64_t(c) * W) : make_int4(0, 0, 0, 0);
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int words[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    acc[i] = __dp4a(words[i >> 2], 1 << (8 * (i & 3)), acc[i]);
                }
            }
        }
    }
    // lanes 4 apart hold the same columns: halve the columns a lane keeps with each exchange
    const int lane = threadIdx.x & 31;
    int first = 0;
#pragma unroll
    for (int half = 8, bit = 4; half >= 2; half >>= 1, bit <<= 1) {
        const bool upper = (lane & bit) != 0;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const int32_t give = upper ? acc[i] : acc[i + half], keep = upper ? acc[i + half] : acc[i];
            acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
        }
        first += upper ? half : 0;
    }
    part[threadIdx.x >> 5][seg * 16 + first] = acc[0];
    part[threadIdx.x >> 5][seg * 16 + first + 1] = acc[1];
    __syncthreads();
    if (threadIdx.x < 64 && w0 + threadIdx.x < W) {
        int32_t sum = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            sum += part[q][threadIdx.x];
        }
        corr[int64_t(n) * W + w0 + threadIdx.x] = int32_t(uint32_t(0) - uint32_t(za) * uint32_t(sum));
    }
}

// ---- AVG_POOL2D, int8 NHWC (avgpool2d.comp:27-75) ---------------------------------------------------------
// One output pixel and up to `width` channel units (a unit is 16 channels, or four or one where C asks for it) belong to a cluster of
// `split` blocks.  The in-range part of a window is rows of contiguous bytes, one run when it spans whole image rows (a
// global pool), so a thread keeps one channel unit and strides over the pixels of its block's share: consecutive threads
// read consecutive bytes whatever the channel count.  Partial sums join in shared memory, first of the block, then of
// the cluster's blocks in block 0 (distributed shared memory).
// The classifier's pool has one output pixel per image: one block for each left the chip idle on small batches and large
// windows (64 images of 112 x 112 x 64: 264 us with one block per pixel, 64 blocks, now 16.6, with 16-byte units, 20.5 with 4-byte ones; a channel count that is no
// multiple of 16 took the one-thread-per-output kernel: 3 x 57 x 57 x 36, 990 us, now 9).
template <int CH>
__global__ void __launch_bounds__(256) avgPoolI8Kernel(const int8_t *__restrict__ in, int8_t *__restrict__ out, int H, int W,
                                                       int C, int OH, int OW, int chunks, int width, int split, PoolAttr a) {
    __shared__ int32_t part[256 * CH];
    const int rank = int(blockIdx.x % unsigned(split));
    unsigned b = blockIdx.x / unsigned(split);
    const int units = C / CH; // per pixel
    const int unit0 = int(b % unsigned(chunks)) * width, unitsHere = min(units - unit0, width);
    b /= unsigned(chunks);
    const int ox = int(b % unsigned(OW));
    b /= unsigned(OW);
    const int oy = int(b % unsigned(OH)), n = int(b / unsigned(OH));
    const int iy = oy * a.stride[0] - a.pad[0], ix = ox * a.stride[1] - a.pad[2];
    const int y0 = max(iy, 0), x0 = max(ix, 0);
    const int ny = max(min(iy + a.kernel[0], H) - y0, 0), nx = max(min(ix + a.kernel[1], W) - x0, 0);
    const int count = ny * nx;

    const int lanes = 256 / unitsHere; // pixels in flight per block
    const int pixel = int(threadIdx.x) / unitsHere, unit = int(threadIdx.x) - pixel * unitsHere;
    int32_t acc[CH];
#pragma unroll
    for (int k = 0; k < CH; ++k) {
        acc[k] = 0;
    }
    if (pixel < lanes) {
        const bool joined = nx == W; // the window's rows follow one another in memory
        const int lines = joined ? 1 : ny, length = joined ? count : nx;
        // this block's share: lines, or a stretch of the one line
        const int line0 = joined ? 0 : int(int64_t(lines) * rank / split), line1 = joined ? 1 : int(int64_t(lines) * (rank + 1) / split);
        const int from = joined ? int(int64_t(length) * rank / split) : 0, to = joined ? int(int64_t(length) * (rank + 1) / split) : length;
        const auto take = [&](const int8_t *p) {
            if (CH == 16) {
                const int4 v = __ldg(reinterpret_cast<const int4 *>(p));
                const int words[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int k = 0; k < CH; ++k) {
                    acc[k] = __dp4a(words[k >> 2], 1 << (8 * (k & 3)), acc[k]);
                }
            } else if (CH == 4) {
                const int word = __ldg(reinterpret_cast<const int *>(p));
#pragma unroll
                for (int k = 0; k < CH; ++k) {
                    acc[k] = __dp4a(word, 1 << (8 * k), acc[k]);
                }
            } else {
                acc[0] += int32_t(__ldg(p));
            }
        };
        for (int line = line0; line < line1; ++line) {
            const int8_t *row = in + ((int64_t(n) * H + y0 + line) * W + x0) * C + (unit0 + unit) * CH;
#pragma unroll 8
            for (int x = from + pixel; x < to; x += lanes) {
                take(row + int64_t(x) * C);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < CH; ++k) {
        part[threadIdx.x * CH + k] = acc[k];
    }
    __syncthreads();
    // sum over the pixels in flight: thread j holds value j of unitsHere * CH
    for (int j = threadIdx.x; j < unitsHere * CH; j += 256) {
        uint32_t v = 0;
        for (int q = 0; q < lanes; ++q) {
            v += uint32_t(part[q * unitsHere * CH + j]);
        }
        part[j] = int32_t(v); // slot j of lane 0 is read by this thread alone
    }
    if (split > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    if (rank == 0) {
        for (int j = threadIdx.x; j < unitsHere * CH; j += 256) {
            uint32_t sum = uint32_t(part[j]);
            for (int r = 1; r < split; ++r) {
                uint32_t peer, v;
                const uint32_t local = uint32_t(__cvta_generic_to_shared(&part[j]));
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(local), "r"(r));
                asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(peer));
                sum += v;
            }
            int32_t v = int32_t(sum - uint32_t(a.inZp) * uint32_t(count));
            if (count == 0) {
                v = 0;
            } else {
                const int32_t round = v < 0 ? -(count >> 1) : (count >> 1);
                v = int32_t(uint32_t(v) + uint32_t(round)) / count; // truncates toward zero
            }
            v = int32_t(uint32_t(v) + uint32_t(a.outZp));
            v = v < -128 ? -128 : (v > 127 ? 127 : v);
            out[((int64_t(n) * OH + oy) * OW + ox) * C + unit0 * CH + j] = int8_t(v);
        }
    }
    if (split > 1) { // block 0 has read the others' shared memory before they leave
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

// ---- MAX_POOL2D, int8 NHWC, C % 16 == 0 (maxpool2d.comp:23-72) --------------------------------------
// One thread per (pixel, 16-channel group): 16-byte loads, per-byte signed max, one 16-byte store.
//
// There is no four-lane byte maximum in hardware, but there is a three-input one on two 16-bit lanes.  A word of
// four int8 is therefore split into its even and its odd bytes, each moved to the HIGH byte of a 16-bit lane with
// a zero below it: the signed order of the lanes is the signed order of the bytes.  One byte permute per half and
// one three-input maximum per half and pair of taps replace the emulated byte maximum.
__device__ __forceinline__ uint32_t evenBytesHigh(uint32_t v) { return __byte_perm(v, 0u, 0x2404); }
__device__ __forceinline__ uint32_t oddBytesHigh(uint32_t v) { return __byte_perm(v, 0u, 0x3414); }
__device__ __forceinline__ uint32_t max3Lanes(uint32_t a, uint32_t b, uint32_t c) { return __vimax3_s16x2(a, b, c); }

struct PoolAcc {
    uint32_t even[4], odd[4];
    __device__ __forceinline__ PoolAcc() {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            even[i] = odd[i] = 0x80008000u; // int8 lowest in both lanes
        }
    }
    __device__ __forceinline__ void take(const int4 &p, const int4 &q) {
        const uint32_t a[4] = {uint32_t(p.x), uint32_t(p.y), uint32_t(p.z), uint32_t(p.w)};
        const uint32_t b[4] = {uint32_t(q.x), uint32_t(q.y), uint32_t(q.z), uint32_t(q.w)};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            even[i] = max3Lanes(even[i], evenBytesHigh(a[i]), evenBytesHigh(b[i]));
            odd[i] = max3Lanes(odd[i], oddBytesHigh(a[i]), oddBytesHigh(b[i]));
        }
    }
    __device__ __forceinline__ void take(const PoolAcc &o) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            even[i] = max3Lanes(even[i], o.even[i], o.even[i]);
            odd[i] = max3Lanes(odd[i], o.odd[i], o.odd[i]);
        }
    }
    __device__ __forceinline__ int4 packed() const {
        // byte 0 and 2 from the high bytes of `even`, byte 1 and 3 from the high bytes of `odd`
        return make_int4(int(__byte_perm(even[0], odd[0], 0x7351)), int(__byte_perm(even[1], odd[1], 0x7351)),
                         int(__byte_perm(even[2], odd[2], 0x7351)), int(__byte_perm(even[3], odd[3], 0x7351)));
    }
};

// KH, KW > 0: the window is known at compile time, all its loads are issued before the first maximum.
// KH == 0: any window, two taps at a time.
template <int KH, int KW>
__global__ void maxPoolI8Kernel(const int8_t *in, int8_t *out, int64_t total, int H, int W,
                                int C, int OH, int OW, PoolAttr a) {
    dependencySync();
    const int groups = C >> 4;
    const int4 lowest = make_int4(int(0x80808080u), int(0x80808080u), int(0x80808080u), int(0x80808080u));
    for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < total; e += int64_t(gridDim.x) * blockDim.x) {
        const int g = int(e % groups);
        int64_t pix = e / groups;
        const int ox = int(pix % OW);
        pix /= OW;
        const int oy = int(pix % OH);
        const int n = int(pix / OH);
        const int iy0 = oy * max(a.stride[0], 1) - a.pad[0], ix0 = ox * max(a.stride[1], 1) - a.pad[2];
        const int4 *image = reinterpret_cast<const int4 *>(in + int64_t(n) * H * W * C) + g;
        const auto tap = [&](int y, int x) {
            return (unsigned(y) < unsigned(H) && unsigned(x) < unsigned(W)) ? image[(int64_t(y) * W + x) * groups]
                                                                            : lowest;
        };
        PoolAcc acc;
        if constexpr (KH > 0) {
            constexpr int kTaps = KH * KW;
            int4 v[kTaps + 1];
#pragma unroll
            for (int t = 0; t < kTaps; ++t) {
                v[t] = tap(iy0 + t / KW, ix0 + t % KW);
            }
            v[kTaps] = lowest;
#pragma unroll
            for (int t = 0; t < kTaps; t += 2) {
                acc.take(v[t], v[t + 1]);
            }
        } else {
            const int taps = a.kernel[0] * a.kernel[1];
            for (int t = 0; t < taps; t += 2) {
                const int4 p = tap(iy0 + t / a.kernel[1], ix0 + t % a.kernel[1]);
                const int4 q = t + 1 < taps ? tap(iy0 + (t + 1) / a.kernel[1], ix0 + (t + 1) % a.kernel[1]) : lowest;
                acc.take(p, q);
            }
        }
        reinterpret_cast<int4 *>(out + ((int64_t(n) * OH + oy) * OW + ox) * C)[g] = acc.packed();
    }
}

// Channel counts that are no multiple of 16: a thread per output pixel and four channels (CH == 4, C % 4 == 0) or one.
template <int CH>
__global__ void __launch_bounds__(256) maxPoolNarrowKernel(const int8_t *in, int8_t *out,
                                                           uint32_t total, int H, int W, int C, FastDiv groups, FastDiv divOW,
                                                           FastDiv divOH, PoolAttr a) {
    dependencySync();
    const uint32_t step = gridDim.x * blockDim.x;
    for (uint64_t e64 = blockIdx.x * blockDim.x + threadIdx.x; e64 < total; e64 += step) {
        const uint32_t e = uint32_t(e64);
        const uint32_t pix = fastDiv(e, groups), line = fastDiv(pix, divOW), n = fastDiv(line, divOH);
        const int c0 = int(e - pix * groups.d) * CH;
        const int ox = int(pix - line * divOW.d), oy = int(line - n * divOH.d);
        const int iy0 = oy * max(a.stride[0], 1) - a.pad[0], ix0 = ox * max(a.stride[1], 1) - a.pad[2];
        const int y0 = max(iy0, 0), y1 = min(iy0 + a.kernel[0], H), x0 = max(ix0, 0), x1 = min(ix0 + a.kernel[1], W);
        const int8_t *image = in + int64_t(n) * H * W * C + c0;
        uint32_t even = 0x80008000u, odd = 0x80008000u; // int8 lowest in both lanes
        int32_t top = -128;
        for (int y = y0; y < y1; ++y) {
#pragma unroll 4
            for (int x = x0; x < x1; ++x) {
                const int8_t *p = image + (int64_t(y) * W + x) * C;
                if (CH == 4) {
                    const uint32_t w = *reinterpret_cast<const uint32_t *>(p);
                    even = max3Lanes(even, evenBytesHigh(w), even);
                    odd = max3Lanes(odd, oddBytesHigh(w), odd);
                } else {
                    top = max(top, int32_t(*p));
                }
            }
        }
        if (CH == 4) {
            reinterpret_cast<uint32_t *>(out)[e] = __byte_perm(even, odd, 0x7351);
        } else {
            out[e] = int8_t(top);
        }
    }
}

// The 3x3 window with stride 2 (the stem pool of the residual networks): one thread makes two horizontally
// adjacent outputs, whose windows share a column, from 15 loads instead of 18.  OW must be even.
__global__ void maxPool3x3s2PairKernel(const int8_t *in, int8_t *out, int64_t total, int H,
                                       int W, int C, int OH, int OW, int padTop, int padLeft) {
    dependencySync();
    const int groups = C >> 4, pairs = OW >> 1;
    const int4 lowest = make_int4(int(0x80808080u), int(0x80808080u), int(0x80808080u), int(0x80808080u));
    for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < total; e += int64_t(gridDim.x) * blockDim.x) {
        const int g = int(e % groups);
        int64_t pix = e / groups;
        const int ox = int(pix % pairs) * 2;
        pix /= pairs;
        const int oy = int(pix % OH);
        const int n = int(pix / OH);
        const int iy0 = oy * 2 - padTop, ix0 = ox * 2 - padLeft;
        const int4 *image = reinterpret_cast<const int4 *>(in + int64_t(n) * H * W * C) + g;
        int4 v[3][5];
#pragma unroll
        for (int ky = 0; ky < 3; ++ky) {
#pragma unroll
            for (int kx = 0; kx < 5; ++kx) {
                const int y = iy0 + ky, x = ix0 + kx;
                v[ky][kx] = (unsigned(y) < unsigned(H) && unsigned(x) < unsigned(W))
                                ? image[(int64_t(y) * W + x) * groups]
                                : lowest;
            }
        }
        PoolAcc left, right, shared;
        shared.take(v[0][2], v[1][2]);
        shared.take(v[2][2], lowest);
#pragma unroll
        for (int ky = 0; ky < 3; ++ky) {
            left.take(v[ky][0], v[ky][1]);
            right.take(v[ky][3], v[ky][4]);
        }
        left.take(shared);
        right.take(shared);
        int4 *o = reinterpret_cast<int4 *>(out + ((int64_t(n) * OH + oy) * OW + ox) * C) + g;
        o[0] = left.packed();
        o[groups] = right.packed();
    }
}

// The same window and stride, a block of 2 x 2 outputs per thread (OH and OW even): the four windows cover 5 x 5
// input pixels, 25 loads instead of 36.  Every pixel word is split into its even and odd byte lanes once; a row
// gives the horizontal maxima of the left and of the right window, which the upper and the lower output share.
struct LaneWords {
    uint32_t even[4], odd[4];
};
__device__ __forceinline__ LaneWords toLanes(const int4 &v) {
    const uint32_t w[4] = {uint32_t(v.x), uint32_t(v.y), uint32_t(v.z), uint32_t(v.w)};
    LaneWords l;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        l.even[i] = evenBytesHigh(w[i]);
        l.odd[i] = oddBytesHigh(w[i]);
    }
    return l;
}
__device__ __forceinline__ LaneWords max3(const LaneWords &a, const LaneWords &b, const LaneWords &c) {
    LaneWords r;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        r.even[i] = max3Lanes(a.even[i], b.even[i], c.even[i]);
        r.odd[i] = max3Lanes(a.odd[i], b.odd[i], c.odd[i]);
    }
    return r;
}
__device__ __forceinline__ int4 packLanes(const LaneWords &l) {
    return make_int4(int(__byte_perm(l.even[0], l.odd[0], 0x7351)), int(__byte_perm(l.even[1], l.odd[1], 0x7351)),
                     int(__byte_perm(l.even[2], l.odd[2], 0x7351)), int(__byte_perm(l.even[3], l.odd[3], 0x7351)));
}

__global__ void maxPool3x3s2QuadKernel(const int8_t *in, int8_t *out, int64_t total, int H,
                                       int W, int C, int OH, int OW, int padTop, int padLeft) {
    dependencySync();
    const int groups = C >> 4, pairsX = OW >> 1, pairsY = OH >> 1;
    const int4 lowest = make_int4(int(0x80808080u), int(0x80808080u), int(0x80808080u), int(0x80808080u));
    for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < total; e += int64_t(gridDim.x) * blockDim.x) {
        const int g = int(e % groups);
        int64_t pix = e / groups;
        const int ox = int(pix % pairsX) * 2;
        pix /= pairsX;
        const int oy = int(pix % pairsY) * 2;
        const int n = int(pix / pairsY);
        const int iy0 = oy * 2 - padTop, ix0 = ox * 2 - padLeft;
        const int4 *image = reinterpret_cast<const int4 *>(in + int64_t(n) * H * W * C) + g;
        LaneWords rowL[5], rowR[5];
#pragma unroll
        for (int ky = 0; ky < 5; ++ky) {
            int4 v[5];
#pragma unroll
            for (int kx = 0; kx < 5; ++kx) {
                const int y = iy0 + ky, x = ix0 + kx;
                v[kx] = (unsigned(y) < unsigned(H) && unsigned(x) < unsigned(W)) ? image[(int64_t(y) * W + x) * groups]
                                                                                 : lowest;
            }
            const LaneWords mid = toLanes(v[2]);
            rowL[ky] = max3(toLanes(v[0]), toLanes(v[1]), mid);
            rowR[ky] = max3(mid, toLanes(v[3]), toLanes(v[4]));
        }
        int4 *o = reinterpret_cast<int4 *>(out + ((int64_t(n) * OH + oy) * OW + ox) * C) + g;
        o[0] = packLanes(max3(rowL[0], rowL[1], rowL[2]));
        o[groups] = packLanes(max3(rowR[0], rowR[1], rowR[2]));
        o[int64_t(OW) * groups] = packLanes(max3(rowL[2], rowL[3], rowL[4]));
        o[int64_t(OW) * groups + groups] = packLanes(max3(rowR[2], rowR[3], rowR[4]));
    }
}

int finish(const char *what) {
    const cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) {
        setLastError(std::string(what) + ": " + cudaGetErrorString(err));
        return MLEL_ERROR_DEVICE;
    }
    return MLEL_SUCCESS;
}

} // namespace

int padImageI8(const int8_t *in, int8_t *out, int N, int H, int W, int C, int Hp, int Wp, int Cp, int padTop, int padLeft,
               cudaStream_t s) {
    if (Cp == 4 && C <= 4 && Wp % 2 == 0 && int64_t(N) * Hp < (int64_t(1) << 31) &&
        (reinterpret_cast<uintptr_t>(out) & 7u) == 0) {
        launchOverlapped(padImageRows4Kernel, dim3(unsigned(N * Hp)), 128, 0, s, in, out, H, W, C, Hp, Wp, padTop, padLeft);
        return finish("padded copy");
    }
    const int64_t pixels = int64_t(N) * Hp * Wp, units = pixels * (Cp >> 4);
    if (Cp % 16 == 0 && units < (int64_t(1) << 30) && (reinterpret_cast<uintptr_t>(out) & 15u) == 0) {
        const bool border = Hp != H || Wp != W || padTop != 0 || padLeft != 0;
        launchOverlapped(border ? padPixels16Kernel<true> : padPixels16Kernel<false>, dim3(gridFor(units, 256, 8)), 256, 0, s,
            in, reinterpret_cast<int4 *>(out), uint32_t(units), H, W, C, makeFastDiv(Cp >> 4), makeFastDiv(Wp), makeFastDiv(Hp), padTop,
            padLeft);
        return finish("padded copy");
    }
    const int64_t words = int64_t(N) * Hp * Wp * (Cp >> 2);
    launchOverlapped(padImageKernel, dim3(gridFor(words, kThreads, 8)), kThreads, 0, s, in, out, words, H, W, C, Hp, Wp, Cp, padTop, padLeft);
    return finish("padded copy");
}

int gatherUnitsI8(const int8_t *in, void *out, int N, int H, int W, int C, int Hu, int Wu, int stride, int padTop, int padLeft,
                  cudaStream_t s) {
    const int64_t units = int64_t(N) * Hu * Wu;
    launchOverlapped(stride == 1 ? gatherUnitsKernel<1> : gatherUnitsKernel<2>, dim3(gridFor(units, 256, 8)), 256, 0, s, in,
                     reinterpret_cast<int4 *>(out), uint32_t(units), H, W, C, makeFastDiv(Wu), makeFastDiv(Hu), padTop, padLeft);
    return finish("units of four pixels");
}

int transposeForMatmul(const int8_t *b, int8_t *bt, int32_t *corr, int batches, int C, int W, int32_t za, cudaStream_t s) {
    // more blocks per 64 columns while the SMs are not filled twice over and each keeps two tiles of rows
    const int columns = (W + 63) / 64, tiles = (C + 63) / 64;
    int split = 1;
    while (split < 8 && int64_t(columns) * batches * split < 2 * kNumSMs && tiles >= 4 * split) {
        split *= 2;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(unsigned(columns * split), unsigned(batches));
    cfg.blockDim = dim3(256);
    cfg.stream = s;
    cudaLaunchAttribute attrs[2]{};
    attrs[0].id = cudaLaunchAttributeClusterDimension;
    attrs[0].val.clusterDim.x = unsigned(split);
    attrs[0].val.clusterDim.y = attrs[0].val.clusterDim.z = 1;
    // A small operand's transpose as a dependent launch (5 x 128 x 160 x 48 8.2 -> 6.5 us a pass).  A large one's blocks would settle
    // beside the product of the pass before, whose shared memory leaves them little of the cache that their loads in flight
    // need (45 x 45 x 864 x 298 24.6 -> 37 us, 6 x 213 x 512 x 570 12.3 -> 16.3).
    attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attrs;
    cfg.numAttrs = dependentLaunches() && int64_t(batches) * C * W <= int64_t(1) << 18 ? 2 : 1;
    cudaLaunchKernelEx(&cfg, W % 16 == 0 ? transposeColsumKernel<true> : transposeColsumKernel<false>, b, bt, corr, C, W,
                       (C + 15) / 16 * 16, za, split);
    return finish("MATMUL operand transpose");
}

int columnSumsForMatmul(const int8_t *b, int32_t *corr, int batches, int C, int W, int32_t za, cudaStream_t s) {
    const dim3 grid(unsigned((W + 63) / 64), unsigned(batches));
    launchOverlapped(columnSumKernel, grid, 256, 0, s, b, corr, C, W, za);
    return finish("MATMUL operand column sums");
}

// Packed int8 NHWC tensors; the kernels look at the channel count and the addresses themselves.
bool poolI8Eligible(const TView &in, const TView &out) {
    const auto packed = [](const TView &t) {
        int64_t s = 1;
        for (int i = t.rank - 1; i >= 0; --i) {
            if (t.strides[i] != s) {
                return false;
            }
            s *= t.dims[i];
        }
        return s > 0 && s < (int64_t(1) << 40);
    };
    return in.dtype == MLEL_I8 && out.dtype == MLEL_I8 && in.rank == 4 && out.rank == 4 && in.dims[3] == out.dims[3] &&
           in.dims[0] == out.dims[0] && packed(in) && packed(out);
}

namespace {
// Widest access (16, 4 or 1 bytes) that the channel count and both addresses allow.
int poolUnit(const TView &in, const TView &out) {
    const uintptr_t bits =
        uintptr_t(in.dims[3]) | reinterpret_cast<uintptr_t>(in.ptr) | reinterpret_cast<uintptr_t>(out.ptr);
    return (bits & 15u) == 0 ? 16 : ((bits & 3u) == 0 ? 4 : 1);
}
} // namespace

bool maxPoolI8Eligible(const TView &in, const TView &out) {
    int64_t n = 1;
    for (int i = 0; i < out.rank; ++i) {
        n *= out.dims[i];
    }
    return poolI8Eligible(in, out) && (poolUnit(in, out) == 16 || n / poolUnit(in, out) < (int64_t(1) << 31));
}

bool avgPoolI8Eligible(const TView &in, const TView &out, const PoolAttr &a) {
    // one block or more per output pixel and 256 channel units: worthwhile when the window is large
    return poolI8Eligible(in, out) && a.kernel[0] > 0 && a.kernel[1] > 0 && int64_t(a.kernel[0]) * a.kernel[1] >= 16 &&
           int64_t(a.kernel[0]) * a.kernel[1] < (int64_t(1) << 24) && a.stride[0] > 0 && a.stride[1] > 0 &&
           int64_t(out.dims[0]) * out.dims[1] * out.dims[2] * ((int64_t(out.dims[3]) + 31) / 32) < (int64_t(1) << 27);
}

int avgPoolI8(const TView &in, const TView &out, const PoolAttr &a, cudaStream_t s) {
    const int C = int(in.dims[3]);
    const int ch = poolUnit(in, out), units = C / ch; // 16, 4 or 1 channels
    const int64_t pixels = int64_t(out.dims[0]) * out.dims[1] * out.dims[2];
    // More blocks while the SMs are not filled four times over: first of fewer channels, down to 128 bytes, so that a
    // block has more pixels in flight; then a cluster per group while a block's share is no less than the 256 threads
    // fetch in one go of eight units (below that the cluster's barriers cost more than the shorter walk
    // gives: 64 images of 7 x 7 x 2048 took 20.4 us as clusters of eight blocks of 256 units).
    int width = 256;
    const int narrowest = ch == 16 ? 8 : 32;
    while (width > narrowest && pixels * ((units + width - 1) / width) < 4 * kNumSMs) {
        width /= 2;
    }
    const int chunks = (units + width - 1) / width;
    const int64_t groups = pixels * chunks;
    const int64_t bytes = int64_t(std::min(a.kernel[0], int(in.dims[1]))) * std::min(a.kernel[1], int(in.dims[2])) *
                          std::min(units, width) * ch;
    int split = 1;
    while (split < 8 && groups * split < 4 * kNumSMs && bytes / (2 * split) >= 256 * 8 * ch) {
        split *= 2;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(unsigned(groups * split));
    cfg.blockDim = dim3(256);
    cfg.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = unsigned(split);
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, ch == 16 ? avgPoolI8Kernel<16> : (ch == 4 ? avgPoolI8Kernel<4> : avgPoolI8Kernel<1>), reinterpret_cast<const int8_t *>(in.ptr),
                       reinterpret_cast<int8_t *>(out.ptr), int(in.dims[1]), int(in.dims[2]), C, int(out.dims[1]),
                       int(out.dims[2]), chunks, width, split, a);
    return finish("AVG_POOL2D");
}

int maxPoolI8(const TView &in, const TView &out, const PoolAttr &a, cudaStream_t s) {
    if (const int unit = poolUnit(in, out); unit < 16) {
        const int64_t words = int64_t(out.dims[0]) * out.dims[1] * out.dims[2] * (out.dims[3] / unsigned(unit));
        const auto kernel = unit == 4 ? maxPoolNarrowKernel<4> : maxPoolNarrowKernel<1>;
        launchOverlapped(kernel, dim3(gridFor(words, kThreads, 16)), kThreads, 0, s, 
            reinterpret_cast<const int8_t *>(in.ptr), reinterpret_cast<int8_t *>(out.ptr), uint32_t(words), int(in.dims[1]),
            int(in.dims[2]), int(in.dims[3]), makeFastDiv(out.dims[3] / unsigned(unit)), makeFastDiv(out.dims[2]),
            makeFastDiv(out.dims[1]), a);
        return finish("MAX_POOL2D");
    }
    const int64_t total = int64_t(out.dims[0]) * out.dims[1] * out.dims[2] * (out.dims[3] >> 4);
    const auto launch = [&](auto kernel) {
        launchOverlapped(kernel, dim3(gridFor(total, kThreads, 16)), kThreads, 0, s, 
            reinterpret_cast<const int8_t *>(in.ptr), reinterpret_cast<int8_t *>(out.ptr), total, int(in.dims[1]),
            int(in.dims[2]), int(in.dims[3]), int(out.dims[1]), int(out.dims[2]), a);
    };
    if (a.kernel[0] == 3 && a.kernel[1] == 3 && a.stride[0] == 2 && a.stride[1] == 2 && out.dims[2] % 2 == 0 &&
        out.dims[1] % 2 == 0) {
        const int64_t quads = total / 4;
        launchOverlapped(maxPool3x3s2QuadKernel, dim3(gridFor(quads, 128, 16)), 128, 0, s, 
            reinterpret_cast<const int8_t *>(in.ptr), reinterpret_cast<int8_t *>(out.ptr), quads, int(in.dims[1]),
            int(in.dims[2]), int(in.dims[3]), int(out.dims[1]), int(out.dims[2]), a.pad[0], a.pad[2]);
    } else if (a.kernel[0] == 3 && a.kernel[1] == 3 && a.stride[0] == 2 && a.stride[1] == 2 && out.dims[2] % 2 == 0) {
        const int64_t pairs = total / 2;
        launchOverlapped(maxPool3x3s2PairKernel, dim3(gridFor(pairs, kThreads, 16)), kThreads, 0, s, 
            reinterpret_cast<const int8_t *>(in.ptr), reinterpret_cast<int8_t *>(out.ptr), pairs, int(in.dims[1]),
            int(in.dims[2]), int(in.dims[3]), int(out.dims[1]), int(out.dims[2]), a.pad[0], a.pad[2]);
    } else if (a.kernel[0] == 3 && a.kernel[1] == 3) {
        launch(maxPoolI8Kernel<3, 3>);
    } else if (a.kernel[0] == 2 && a.kernel[1] == 2) {
        launch(maxPoolI8Kernel<2, 2>);
    } else {
        launch(maxPoolI8Kernel<0, 0>);
    }
    return finish("MAX_POOL2D");
}

} // namespace mlel
