// DEPTHWISE_CONV2D 3x3 + RESCALE (+CLAMP) on int8 NHWC tensors of any channel count, from a table of per-channel constants
// (depthwise_conv2d.comp:31-78, rescale.comp:27-72).
//
// A thread owns four channels of a block of 4 output pixels x R output rows.  Input rows stream through once: a row's pixel
// words are transposed four at a time (4 pixels x 4 channels -> 4 channels x 4 pixels, eight byte-permutes), so that three
// neighbouring taps of one channel lie in one word; one dp4a against the channel's three weights of that window row (at byte
// offset 0 or 1, for the windows that start at the word's first and second pixel) gives three multiply-accumulates.  An input
// row feeds the up to three output rows whose windows contain it.  Out-of-range taps read the input zero point, and what the
// zero point contributes is in the constants.
//
// Bound by the instructions it issues, not by memory.  What the kernel without the table (depthwise3x3RowsKernel, which
// remains for what a table does not describe) spends beside three dp4a, one and a half byte-permutes and the product of the
// RESCALE: three instructions an output (six with R = 2) on packing weights and building RESCALE constants, which are graph
// constants and made by the host here; sums start at bias, zero points and all, so that the sign which double rounding asks for
// is the sum's own, and the addend takes it in two instructions with the output zero point inside; results are packed
// saturating, so that bounds at the ends of the range cost nothing.
//
// Channel counts that are no multiple of four: the words start at any byte and are joined from two aligned ones, results leave
// byte by byte.
//
// The table stands word by word for all groups of channels, not channel by channel: neighbouring threads have neighbouring groups, and
// with 128 bytes between their words each of a thread's eight loads of it took a warp 32 lines, 2 us of an SM with 16 warps.  (32 x 28 x
// 28 x 192 7.9 us without the table, 8.7 so, 5.6 now; 32 x 14 x 14 x 576 7.1, 8.7 and 5.0; 32 images of the MobileNetV2 shape 450 -> 418.)
//
// Measured (us, without the table -> now): 64 x 112 x 112 x 64 59.8 -> 43.1, with a ReLU 53.7 -> 41.4; 32 x 56 x 56 x 144 17.2 -> 13.1;
// 63 channels (one thread per output before) 2244 -> 76.5, 16 x 57 x 57 x 35 86 -> 9.3.  Of 16 instructions an output four address its
// loads: a copy of the tile in shared memory would save those.
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "depthwise_i8.hpp"
#include "device_common.cuh"
#include "launch_overlapped.cuh"

namespace mlel {

namespace {

struct DepthwiseParams {
    const int8_t *in;
    int8_t *out;
    const int4 *table; // [8][groups of four channels]
    int32_t N, H, W, C, OH, OW;
    FastDiv divC, divX, divY; // groups of channels, pixels and rows
    int32_t padTop, padLeft;
    uint32_t zeroWord;
    int32_t lo, hi, signedRounding;
};

// The first `bytes` bytes from any address (the others: anything).  Only aligned words that hold one of them are read.
__device__ __forceinline__ uint32_t loadBytes(const int8_t *p, int bytes) {
    const uintptr_t at = reinterpret_cast<uintptr_t>(p);
    const uint32_t skip = uint32_t(at & 3u);
    const uint32_t *words = reinterpret_cast<const uint32_t *>(at - skip);
    const uint32_t first = words[0], second = int(skip) + bytes > 4 ? words[1] : 0u;
    return __funnelshift_r(first, second, 8 * skip);
}

// (x * mult + addend) >> 32 >> shift as bytes of four channels.  SIGNED: the addend is that of x >= 0, a negative x takes 2^31 off
// it: the low word, 2^30 (see makeDepthwiseChannels), changes its top bit and the high word loses one.
template <bool SIGNED, bool BOUNDED>
__device__ __forceinline__ uint32_t rescaleFour(const int32_t (&x)[4], const int4 (&k)[4], int32_t lo, int32_t hi) {
    int32_t y[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        // {low, high, mult, shift}
        const uint32_t low = SIGNED ? uint32_t(k[j].x) ^ (uint32_t(x[j]) & 0x80000000u) : uint32_t(k[j].x);
        const uint32_t high = SIGNED ? uint32_t(k[j].y + (x[j] >> 31)) : uint32_t(k[j].y);
        const uint64_t sum = uint64_t(int64_t(x[j]) * int64_t(k[j].z)) + ((uint64_t(high) << 32) | uint64_t(low));
        y[j] = int32_t(uint32_t(sum >> 32)) >> k[j].w;
        if (BOUNDED) {
            y[j] = min(max(y[j], lo), hi);
        } else if (!SIGNED) {
            y[j] = max(y[j], lo);
        }
    }
    return packSatS8(y[0], y[1], y[2], y[3]);
}

// R: output rows of a thread; SX: stride; ALIGNED: whole words (C, and both tensors' addresses, multiples of four).
template <int R, int SX, bool ALIGNED>
__global__ void __launch_bounds__(128, 4) depthwise3x3TableKernel(const __grid_constant__ DepthwiseParams p) {
    constexpr int PX = 4;
    constexpr int COLS = (PX - 1) * SX + 3; // input pixels under the four windows of a row: 6 or 9
    constexpr int NT = SX == 1 ? 2 : 4;     // transposed groups of four pixels per input row
    constexpr int ROWS = (R - 1) * SX + 3;  // input rows under the R windows of a column
    // Scheduled while the launch before drains, and lets the one after do the same: no activation before the wait.  (Some thread has
    // work and waits: a dimension of 0 is refused when a tensor is declared.)
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int64_t total = int64_t(p.N) * p.divY.d * p.divX.d * p.divC.d;
    for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < total; e += int64_t(gridDim.x) * blockDim.x) {
        const uint32_t tx = fastDiv(uint32_t(e), p.divC), ty = fastDiv(tx, p.divX), tn = fastDiv(ty, p.divY);
        const int c0 = int(uint32_t(e) - tx * p.divC.d) * 4, ox0 = int(tx - ty * p.divX.d) * PX, oy0 = int(ty - tn * p.divY.d) * R;
        const int n = int(tn), bytes = ALIGNED ? 4 : min(4, p.C - c0);
        const int4 *channel = p.table + (uint32_t(e) - tx * p.divC.d); // word 2 k + h: channel[(2 k + h) * groups]
        uint32_t wa[3][4], wb[3][4]; // a window row's three weights at byte offsets 0 and 1
        int32_t acc[R][PX][4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int4 v = __ldg(channel + 2 * k * p.divC.d);
            wa[0][k] = uint32_t(v.x), wa[1][k] = uint32_t(v.y), wa[2][k] = uint32_t(v.z);
#pragma unroll
            for (int ky = 0; ky < 3; ++ky) {
                wb[ky][k] = wa[ky][k] << 8;
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
#pragma unroll
                for (int px = 0; px < PX; ++px) {
                    acc[r][px][k] = v.w;
                }
            }
        }
        asm volatile("griddepcontrol.wait;" ::: "memory"); // (a no-op from the second time on)
        const int x0 = ox0 * SX - p.padLeft, yFirst = oy0 * SX - p.padTop;
        // No range tests where all windows lie inside.
        const auto convolve = [&](auto insideTag) {
            constexpr bool INSIDE = decltype(insideTag)::value;
            const int8_t *row = p.in + (int64_t((n * p.H + yFirst) * p.W + x0) * p.C + c0);
            const auto loadRow = [&](int iy, uint32_t (&cols)[COLS]) {
                const bool rowOk = INSIDE || (yFirst + iy >= 0 && yFirst + iy < p.H);
                const int8_t *at = row;
#pragma unroll
                for (int i = 0; i < COLS; ++i) {
                    const bool ok = INSIDE || (rowOk && x0 + i >= 0 && x0 + i < p.W);
                    cols[i] = !ok ? p.zeroWord : (ALIGNED ? *reinterpret_cast<const uint32_t *>(at) : loadBytes(at, bytes));
                    at += p.C;
                }
                row += p.W * p.C;
            };
            // Two output rows leave registers for all input rows: every load of a thread in flight at once.
            uint32_t all[R == 2 ? ROWS : 1][COLS];
            if (R == 2) {
#pragma unroll
                for (int iy = 0; iy < ROWS; ++iy) {
                    loadRow(iy, all[iy]);
                }
            }
#pragma unroll
            for (int iy = 0; iy < ROWS; ++iy) {
                uint32_t(&cols)[COLS] = all[R == 2 ? iy : 0];
                if (R != 2) {
                    loadRow(iy, cols);
                }
                // tr[g][k]: four consecutive pixels of channel k.  Stride 1: pixels 0-3 and 2-5; window px starts at byte
                // px & 1 of group px >> 1.  Stride 2: pixels 0-3, 2-5, 4-7, 5-8; windows start at bytes 0, 0, 0, 1.
                uint32_t tr[NT][4];
                transpose4x4Bytes(cols[0], cols[1], cols[2], cols[3], tr[0]);
                transpose4x4Bytes(cols[2], cols[3], cols[4], cols[5], tr[1]);
                if (SX == 2) {
                    transpose4x4Bytes(cols[4], cols[5], cols[6], cols[7], tr[2]);
                    transpose4x4Bytes(cols[5], cols[6], cols[7], cols[8], tr[3]);
                }
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int ky = iy - r * SX; // this input row as a row of output row r's window (a compile-time value)
                    if (ky >= 0 && ky < 3) {
#pragma unroll
                        for (int px = 0; px < PX; ++px) {
                            const int g = SX == 1 ? px >> 1 : px;
                            const bool second = SX == 1 ? (px & 1) != 0 : px == 3;
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                const uint32_t weights = second ? wb[ky][k] : wa[ky][k];
                                acc[r][px][k] = __dp4a(int32_t(tr[g][k]), int32_t(weights), acc[r][px][k]);
                            }
                        }
                    }
                }
            }
        };
        // (R == 2 is for small images, where most warps would run both forms one after the other)
        if (R == 4 && x0 >= 0 && x0 + COLS <= p.W && yFirst >= 0 && yFirst + ROWS <= p.H) {
            convolve(std::true_type{});
        } else {
            convolve(std::false_type{});
        }
        int4 scale[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            scale[k] = __ldg(channel + (2 * k + 1) * p.divC.d);
        }
        const bool full = oy0 + R <= p.OH && ox0 + PX <= p.OW;
        const auto finish = [&](auto signedTag, auto boundedTag) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                int8_t *to = p.out + (int64_t((n * p.OH + oy0 + r) * p.OW + ox0) * p.C + c0);
#pragma unroll
                for (int px = 0; px < PX; ++px) {
                    if (full || (oy0 + r < p.OH && ox0 + px < p.OW)) {
                        const uint32_t word = rescaleFour<decltype(signedTag)::value, decltype(boundedTag)::value>(acc[r][px], scale, p.lo, p.hi);
                        if (ALIGNED) {
                            *reinterpret_cast<uint32_t *>(to) = word;
                        } else {
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                if (k < bytes) {
                                    to[k] = int8_t(word >> (8 * k));
                                }
                            }
                        }
                    }
                    to += p.C;
                }
            }
        };
        const bool bounded = p.hi < 127 || (p.signedRounding != 0 && p.lo > -128);
        if (p.signedRounding != 0) {
            bounded ? finish(std::true_type{}, std::true_type{}) : finish(std::true_type{}, std::false_type{});
        } else {
            bounded ? finish(std::false_type{}, std::true_type{}) : finish(std::false_type{}, std::false_type{});
        }
    }
}

} // namespace

bool makeDepthwiseChannels(const DepthwiseConstants &d, std::vector<DepthwiseWord> *out) {
    const size_t groups = size_t(d.channels + 3) / 4;
    const bool signFree = !d.doubleRound || d.lo >= d.outZp;
    out->assign(8 * groups, DepthwiseWord{});
    for (int c = 0; c < d.channels; ++c) {
        DepthwiseChannel k{};
        const int32_t mult = d.mult[d.perChannel ? c : 0], shift = d.shift[d.perChannel ? c : 0];
        int64_t sum = 0;
        for (int ky = 0; ky < 3; ++ky) {
            uint32_t word = 0;
            for (int kx = 0; kx < 3; ++kx) {
                const int8_t w = d.weights[(ky * 3 + kx) * d.channels + c];
                word |= uint32_t(uint8_t(w)) << (8 * kx);
                sum += w;
            }
            k.weights[ky] = word;
        }
        // nine products are at most 9 * 2^14 in size: nothing leaves int32
        const int64_t add = int64_t(d.bias[d.biasCount == 1 ? 0 : c]) - int64_t(d.inputZp) * sum, start = add - d.rescaleZp;
        constexpr int64_t kReach = int64_t(1) << 30;
        // the high word of the sum holds the result from a shift of 32 on; the sign's 2^31 is the low word's top bit from 33 on
        if (std::llabs(add) >= kReach || std::llabs(start) >= kReach || shift < (signFree ? 32 : 33) || shift > 50 || mult < 0) {
            return false;
        }
        const int64_t addend = (int64_t(1) << (shift - 1)) + (d.doubleRound ? int64_t(1) << 30 : 0) + int64_t(d.outZp) * (int64_t(1) << shift);
        k.start = int32_t(start), k.mult = mult, k.shift = shift - 32;
        k.low = uint32_t(uint64_t(addend)), k.high = uint32_t(uint64_t(addend) >> 32);
        for (size_t half = 0; half < 2; ++half) {
            std::memcpy(&(*out)[(2 * size_t(c % 4) + half) * groups + size_t(c / 4)], reinterpret_cast<const DepthwiseWord *>(&k) + half,
                        sizeof(DepthwiseWord));
        }
    }
    return true;
}

bool depthwiseTableTakes(const TView &in, const TView &out, const ConvAttr &a) {
    const auto numel = [](const TView &t) { return int64_t(t.dims[0]) * t.dims[1] * t.dims[2] * t.dims[3]; };
    return a.wZp == 0 && a.dilation[0] == 1 && a.dilation[1] == 1 && a.stride[0] == a.stride[1] && (a.stride[0] == 1 || a.stride[0] == 2) &&
           numel(in) < (int64_t(1) << 31) && numel(out) < (int64_t(1) << 31);
}

int depthwiseFromTable(const TView &in, const TView &table, const TView &out, const ConvAttr &a, const DevRescale &r, cudaStream_t s) {
    DepthwiseParams p{};
    p.in = reinterpret_cast<const int8_t *>(in.ptr), p.out = reinterpret_cast<int8_t *>(out.ptr);
    p.table = reinterpret_cast<const int4 *>(table.ptr);
    p.N = int(in.dims[0]), p.H = int(in.dims[1]), p.W = int(in.dims[2]), p.C = int(in.dims[3]), p.OH = int(out.dims[1]), p.OW = int(out.dims[2]);
    p.padTop = a.pad[0], p.padLeft = a.pad[2];
    p.zeroWord = uint32_t(uint8_t(a.inZp)) * 0x01010101u;
    p.lo = r.lo, p.hi = r.hi;
    p.signedRounding = r.doubleRound != 0 && r.lo < r.outZp;
    constexpr int PX = 4;
    const int groupsX = (p.OW + PX - 1) / PX, groupsC = (p.C + 3) / 4;
    // four output rows a thread unless that leaves SMs without work
    const bool four = int64_t(p.N) * ((p.OH + 3) / 4) * groupsX * groupsC >= int64_t(kNumSMs) * 128 * 4;
    const int groupsY = (p.OH + (four ? 3 : 1)) / (four ? 4 : 2);
    p.divC = makeFastDiv(groupsC), p.divX = makeFastDiv(groupsX), p.divY = makeFastDiv(groupsY);
    const int grid = gridFor(int64_t(p.N) * groupsY * groupsX * groupsC, 128, 16);
    const bool aligned = p.C % 4 == 0 && ((reinterpret_cast<uintptr_t>(p.in) | reinterpret_cast<uintptr_t>(p.out)) & 3u) == 0;
    const auto launch = [&](auto whole, auto bytes) { return launchOverlapped(aligned ? whole : bytes, grid, 128, 0, s, p); };
    const cudaError_t err = a.stride[0] == 1 ? (four ? launch(depthwise3x3TableKernel<4, 1, true>, depthwise3x3TableKernel<4, 1, false>)
                                                     : launch(depthwise3x3TableKernel<2, 1, true>, depthwise3x3TableKernel<2, 1, false>))
                                             : (four ? launch(depthwise3x3TableKernel<4, 2, true>, depthwise3x3TableKernel<4, 2, false>)
                                                     : launch(depthwise3x3TableKernel<2, 2, true>, depthwise3x3TableKernel<2, 2, false>));
    if (err != cudaSuccess) {
        setLastError(std::string("DEPTHWISE_CONV2D 3x3: ") + cudaGetErrorString(err));
        return MLEL_ERROR_DEVICE;
    }
    return MLEL_SUCCESS;
}

} // namespace mlel
