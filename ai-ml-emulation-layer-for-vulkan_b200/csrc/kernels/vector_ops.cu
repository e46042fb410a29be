// Vectorised kernels for the element-wise, table, reduction and data-movement operators on packed
// tensors.  Each has a generic counterpart in generic_ops.cu that defines the result for every rank, stride
// and type; these take the common case - contiguous tensors, signed integer types, operands of the same
// shape or broadcast along the last axis - and move 16 bytes a thread and access where they can, several accesses in
// flight, without index unravelling; reductions have a warp per row.  Where the arithmetic is not the generic kernels'
// own function (RESCALE as one multiply-add, CLAMP on 16-bit lanes, TABLE from words that hold two entries) it gives the
// same bits.  Element counts that are no multiple of a thread's group leave one to fifteen elements, which a thread each
// takes (REDUCE_SUM over 2364 rows of 197 in the one-thread-per-row generic kernel: 132 us, here 6.1; SUB by rows of 197:
// 16.4 -> 6.1 us).
//
// Every entry point returns false when it does not apply; the caller then runs the generic kernel.
#include <algorithm>
#include <string>

#include "device_common.cuh"
#include "gemm_i8_tcgen05.hpp"
#include "kernels.hpp"
#include "launch_overlapped.cuh"

namespace mlel {

namespace {

#define GRID_STRIDE(e, total)                                                                                          \
    for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < (total); e += int64_t(gridDim.x) * blockDim.x)

int finish(const char *what) {
    const cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) {
        setLastError(std::string(what) + ": " + cudaGetErrorString(err));
        return MLEL_ERROR_DEVICE;
    }
    return MLEL_SUCCESS;
}

// Number of elements of a contiguous (byte strides = packed) tensor, or -1.
int64_t packedNumel(const TView &t) {
    int64_t st = dtypeSize(t.dtype), n = 1;
    for (int i = t.rank - 1; i >= 0; --i) {
        if (t.strides[i] != st) {
            return -1;
        }
        st *= t.dims[i];
        n *= t.dims[i];
    }
    return n;
}

bool sameShape(const TView &a, const TView &b) {
    if (a.rank != b.rank) {
        return false;
    }
    for (int i = 0; i < a.rank; ++i) {
        if (a.dims[i] != b.dims[i]) {
            return false;
        }
    }
    return true;
}

// b has out's shape except for a last axis of 1 (one value per row of out).
bool rowBroadcast(const TView &b, const TView &out) {
    if (b.rank != out.rank || out.rank < 1 || b.dims[b.rank - 1] != 1) {
        return false;
    }
    for (int i = 0; i + 1 < out.rank; ++i) {
        if (b.dims[i] != out.dims[i]) {
            return false;
        }
    }
    return true;
}

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

bool signedInt(int32_t dtype) { return dtype == MLEL_I8 || dtype == MLEL_I16 || dtype == MLEL_I32; }

// Four consecutive elements of a signed integer type, widened to int32.
template <typename T> __device__ __forceinline__ void load4(const T *p, int32_t (&v)[4]);
template <> __device__ __forceinline__ void load4<int8_t>(const int8_t *p, int32_t (&v)[4]) {
    const uint32_t w = *reinterpret_cast<const uint32_t *>(p);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        v[k] = int32_t(int8_t(w >> (8 * k)));
    }
}
template <> __device__ __forceinline__ void load4<int16_t>(const int16_t *p, int32_t (&v)[4]) {
    const uint2 w = *reinterpret_cast<const uint2 *>(p);
    v[0] = int32_t(int16_t(w.x)), v[1] = int32_t(int16_t(w.x >> 16));
    v[2] = int32_t(int16_t(w.y)), v[3] = int32_t(int16_t(w.y >> 16));
}
template <> __device__ __forceinline__ void load4<int32_t>(const int32_t *p, int32_t (&v)[4]) {
    const int4 w = *reinterpret_cast<const int4 *>(p);
    v[0] = w.x, v[1] = w.y, v[2] = w.z, v[3] = w.w;
}
// Stores the low bits of four values (the caller has clamped or wants the wrap).
template <typename T> __device__ __forceinline__ void store4(T *p, const int32_t (&v)[4]);
template <> __device__ __forceinline__ void store4<int8_t>(int8_t *p, const int32_t (&v)[4]) {
    *reinterpret_cast<uint32_t *>(p) = uint32_t(uint8_t(v[0])) | (uint32_t(uint8_t(v[1])) << 8) |
                                       (uint32_t(uint8_t(v[2])) << 16) | (uint32_t(uint8_t(v[3])) << 24);
}
template <> __device__ __forceinline__ void store4<int16_t>(int16_t *p, const int32_t (&v)[4]) {
    *reinterpret_cast<uint2 *>(p) = make_uint2(uint32_t(uint16_t(v[0])) | (uint32_t(uint16_t(v[1])) << 16),
                                               uint32_t(uint16_t(v[2])) | (uint32_t(uint16_t(v[3])) << 16));
}
template <> __device__ __forceinline__ void store4<int32_t>(int32_t *p, const int32_t (&v)[4]) {
    *reinterpret_cast<int4 *>(p) = make_int4(v[0], v[1], v[2], v[3]);
}

template <typename T> __host__ __device__ constexpr int32_t lowestOf() {
    return sizeof(T) == 1 ? -128 : (sizeof(T) == 2 ? -32768 : int32_t(0x80000000u));
}
template <typename T> __host__ __device__ constexpr int32_t highestOf() {
    return sizeof(T) == 1 ? 127 : (sizeof(T) == 2 ? 32767 : 0x7fffffff);
}

// A thread's share of `groups`, four at a time while there are four: `load(g)` fetches, `store(g, value)` computes and
// writes; the four loads are issued before the first result (one load at a time left a quarter of the bandwidth unused).
template <typename T, typename LOAD, typename STORE> __device__ __forceinline__ void fourInFlight(int64_t groups, const LOAD &load, const STORE &store) {
    const int64_t step = int64_t(gridDim.x) * blockDim.x;
    int64_t g = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    for (; g + 3 * step < groups; g += 4 * step) {
        T v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[k] = load(g + k * step);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            store(g + k * step, v[k]);
        }
    }
    for (; g < groups; g += step) {
        store(g, load(g));
    }
}

// ---- RESCALE (rescale.comp:27-72) -------------------------------------------------------------------------
// A warp takes blocks of 128 Q elements: a lane has Q groups of four consecutive ones, groups 32 apart, so that every load
// and store of the warp is one run of bytes; all loads are issued before the first result is computed.  (With a lane's
// groups side by side a load touched 32 lines for 16 bytes each.)  What the blocks leave goes four elements or one at a
// time.  FORM: 0 fastRescale, 1 and 2 WordsScale with and without the sign (per-tensor scales; picked by each thread, the
// scale is in device memory).  192 x 384 x 384 int32 -> int8: 32.8 us, now 28.6.
//
// Only int8 results have the zero point in WordsScale's addend: 2^7 times 2^50 leaves room for the product (2^62).  An
// int16 zero point would not from a shift of 48 on, an int32 one of 100 000 from 46 on; there it is added to the result.
template <typename OUT> constexpr bool foldsZeroPoint = sizeof(OUT) == 1;

template <int FORM, typename OUT>
__device__ __forceinline__ void rescaleFour(const int32_t (&v)[4], int32_t (&r)[4], FastRescale f, const WordsScale &words,
                                            const int32_t *mult, const int8_t *shift, int perChannel, int c0, int C, int32_t inZp,
                                            int32_t outZp, int doubleRound) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (FORM != 0) {
            int32_t q = wordsScale<FORM == 1>(words, v[k]);
            if (FORM == 1 || !foldsZeroPoint<OUT>) {
                q = int32_t(uint32_t(q) + uint32_t(outZp)); // 32-bit wrap, as fastRescale
            }
            r[k] = min(max(q, lowestOf<OUT>()), highestOf<OUT>());
            continue;
        }
        if (perChannel) {
            const int c = c0 + k < C ? c0 + k : c0 + k - C; // C >= 4: a group wraps once at most
            f = makeFastRescale(__ldg(mult + c), int32_t(__ldg(shift + c)), inZp, doubleRound != 0);
        }
        r[k] = fastRescale(f, v[k], outZp, lowestOf<OUT>(), highestOf<OUT>());
    }
}

template <int FORM, typename IN, typename OUT>
__device__ __forceinline__ void rescaleBlocks(const IN *__restrict__ in, OUT *__restrict__ out, int64_t blocks, const FastRescale &f,
                                              const WordsScale &words, const int32_t *mult, const int8_t *shift, int perChannel,
                                              int C, int32_t inZp, int32_t outZp, int doubleRound) {
    constexpr int Q = 4;
    const int lane = int(threadIdx.x & 31u);
    const int64_t warps = (int64_t(gridDim.x) * blockDim.x) >> 5;
    for (int64_t b = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; b < blocks; b += warps) {
        const int64_t e0 = b * (128 * Q) + lane * 4;
        int32_t v[Q][4];
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            load4<IN>(in + e0 + 128 * q, v[q]);
        }
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            int32_t r[4];
            const int c0 = perChannel ? int((e0 + 128 * q) % C) : 0;
            rescaleFour<FORM, OUT>(v[q], r, f, words, mult, shift, perChannel, c0, C, inZp, outZp, doubleRound);
            store4<OUT>(out + e0 + 128 * q, r);
        }
    }
}

template <typename IN, typename OUT>
__global__ void rescaleVecKernel(const IN *__restrict__ in, OUT *__restrict__ out, int64_t blocks, int64_t tailGroups, int rest,
                                 const int32_t *__restrict__ mult, const int8_t *__restrict__ shift, int perChannel, int C,
                                 int32_t inZp, int32_t outZp, int doubleRound) {
    const FastRescale f = makeFastRescale(__ldg(mult), int32_t(__ldg(shift)), inZp, doubleRound != 0);
    const int s = f.s1 + f.s2;
    WordsScale words{};
    // (a value minus the zero point has to stay inside int32)
    if (!perChannel && wordsScaleApplies(f.mult, s, doubleRound != 0) && (sizeof(IN) < 4 || inZp == 0)) {
        if (doubleRound != 0) {
            words = makeWordsScale<true>(f.mult, s, true, int32_t(uint32_t(0) - uint32_t(inZp)), 0);
            rescaleBlocks<1, IN, OUT>(in, out, blocks, f, words, mult, shift, 0, C, inZp, outZp, doubleRound);
        } else {
            words = makeWordsScale<false>(f.mult, s, false, int32_t(uint32_t(0) - uint32_t(inZp)), foldsZeroPoint<OUT> ? outZp : 0);
            rescaleBlocks<2, IN, OUT>(in, out, blocks, f, words, mult, shift, 0, C, inZp, outZp, doubleRound);
        }
    } else {
        rescaleBlocks<0, IN, OUT>(in, out, blocks, f, words, mult, shift, perChannel, C, inZp, outZp, doubleRound);
    }
    GRID_STRIDE(g, tailGroups + rest) {
        if (g < tailGroups) {
            const int64_t e0 = blocks * 512 + g * 4;
            int32_t v[4], r[4];
            load4<IN>(in + e0, v);
            rescaleFour<0, OUT>(v, r, f, words, mult, shift, perChannel, perChannel ? int(e0 % C) : 0, C, inZp, outZp, doubleRound);
            store4<OUT>(out + e0, r);
        } else { // the last one to three elements, a thread each
            const int64_t e = blocks * 512 + tailGroups * 4 + (g - tailGroups);
            FastRescale fe = f;
            if (perChannel) {
                fe = makeFastRescale(__ldg(mult + e % C), int32_t(__ldg(shift + e % C)), inZp, doubleRound != 0);
            }
            out[e] = OUT(fastRescale(fe, int32_t(in[e]), outZp, lowestOf<OUT>(), highestOf<OUT>()));
        }
    }
}

template <typename IN, typename OUT>
void launchRescale(const TView &in, const TView &out, const TView &mult, const TView &shift, const RescaleAttr &a,
                   int64_t n, cudaStream_t s) {
    const int C = int(out.dims[out.rank - 1]);
    // blocks of 512 elements where every SM gets eight warps of them; below that more threads with fewer elements
    const int64_t blocks = n >= int64_t(512) * kNumSMs * 8 ? n / 512 : 0, tailGroups = (n - blocks * 512) / 4;
    const int64_t threads = blocks != 0 ? blocks * 32 : tailGroups + n % 4;
    rescaleVecKernel<IN, OUT><<<gridFor(threads, kThreads, 16), kThreads, 0, s>>>(
        reinterpret_cast<const IN *>(in.ptr), reinterpret_cast<OUT *>(out.ptr), blocks, tailGroups, int(n % 4),
        reinterpret_cast<const int32_t *>(mult.ptr), reinterpret_cast<const int8_t *>(shift.ptr), a.perChannel ? 1 : 0, C,
        int32_t(wrapTo(in.dtype, a.inZp)), int32_t(wrapTo(out.dtype, a.outZp)), (a.scale32 && a.doubleRound) ? 1 : 0);
}

// ---- TABLE (table.comp:17-52) -------------------------------------------------------------------------------
__global__ void tableI8Kernel(const int8_t *in, int8_t *out, int64_t groups, int rest, const int8_t *table) {
    dependencySync();
    __shared__ int8_t lut[256];
    for (int i = threadIdx.x; i < 256; i += blockDim.x) {
        lut[i] = table[i];
    }
    __syncthreads();
    GRID_STRIDE(g, groups + rest) {
        if (g >= groups) { // the last elements, a thread each
            const int64_t e = 16 * groups + (g - groups);
            out[e] = lut[int(in[e]) + 128];
            continue;
        }
        const int4 w = *reinterpret_cast<const int4 *>(in + 16 * g);
        const uint32_t words[4] = {uint32_t(w.x), uint32_t(w.y), uint32_t(w.z), uint32_t(w.w)};
        uint32_t res[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            uint32_t r = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int idx = int(int8_t(words[q] >> (8 * k))) + 128;
                r |= uint32_t(uint8_t(lut[idx])) << (8 * k);
            }
            res[q] = r;
        }
        *reinterpret_cast<int4 *>(out + 16 * g) = make_int4(int(res[0]), int(res[1]), int(res[2]), int(res[3]));
    }
}

// Large tensors: a copy of the table per lane of a warp, entry b of lane l in word 32 b + l, so that a warp's 32 lookups
// never meet in a bank.  In one table of 64 words they queue up three and a half deep, which bound the kernel (64 x 112 x
// 112 x 64 24.5 us, now 23.2); the 32 KB to fill first are worth it from a few megabytes on.
constexpr int kLaneTableThreads = 1024;
__global__ void __launch_bounds__(kLaneTableThreads) tableI8LanesKernel(const int8_t *__restrict__ in, int8_t *__restrict__ out,
                                                                        int64_t groups, int rest, const int8_t *__restrict__ table) {
    __shared__ uint32_t lanes[256 * 32];
    const uint32_t lane = threadIdx.x & 31u;
    for (int b = int(threadIdx.x >> 5); b < 256; b += kLaneTableThreads / 32) { // raw byte b: value int8(b)
        lanes[b * 32 + int(lane)] = uint32_t(uint8_t(__ldg(table + (b ^ 128))));
    }
    __syncthreads();
    const uint32_t base = uint32_t(__cvta_generic_to_shared(lanes)) + lane * 4u;
    const auto look = [&](uint32_t b128) { // byte times 128
        uint32_t v;
        asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(base + b128));
        return v;
    };
    const auto four = [&](uint32_t w) {
        const uint32_t v0 = look((w << 7) & 0x7f80u), v1 = look((w >> 1) & 0x7f80u), v2 = look((w >> 9) & 0x7f80u),
                       v3 = look((w >> 17) & 0x7f80u);
        return __byte_perm(__byte_perm(v0, v1, 0x0040), __byte_perm(v2, v3, 0x0040), 0x5410);
    };
    fourInFlight<uint4>(
        groups, [&](int64_t g) { return *reinterpret_cast<const uint4 *>(in + 16 * g); },
        [&](int64_t g, const uint4 &w) {
            *reinterpret_cast<uint4 *>(out + 16 * g) = make_uint4(four(w.x), four(w.y), four(w.z), four(w.w));
        });
    GRID_STRIDE(g, rest) { // the last elements, a thread each
        const int64_t e = 16 * groups + g;
        out[e] = int8_t(look(uint32_t(uint8_t(in[e])) * 128u));
    }
}

__device__ __forceinline__ int32_t interpolateI16(const int16_t *lut, int32_t v) {
    const int32_t index = (v + 32768) >> 7;
    const int32_t fraction = v & 0x7f;
    const int32_t base = lut[index], next = lut[index + 1];
    return int32_t((uint32_t(base) << 7) + uint32_t(next - base) * uint32_t(fraction));
}

// The same from words that hold an entry and its successor: one shared-memory read per element (the reads' bank conflicts
// bound the kernel: 192 x 384 x 384 41.0 us, now 29.7).
__device__ __forceinline__ int32_t interpolatePair(const uint32_t *pairs, int32_t v) {
    const uint32_t pair = pairs[(v + 32768) >> 7];
    const int32_t base = int32_t(int16_t(pair)), next = int32_t(pair) >> 16;
    return int32_t((uint32_t(base) << 7) + uint32_t(next - base) * uint32_t(v & 0x7f));
}

__global__ void tableI16Kernel(const int16_t *__restrict__ in, int32_t *__restrict__ out, int64_t groups, int rest,
                               const int16_t *__restrict__ table) {
    __shared__ uint32_t pairs[512];
    for (int i = threadIdx.x; i < 512; i += blockDim.x) {
        pairs[i] = uint32_t(uint16_t(table[i])) | (uint32_t(uint16_t(table[i + 1])) << 16);
    }
    __syncthreads();
    fourInFlight<uint2>(
        groups, [&](int64_t g) { return *reinterpret_cast<const uint2 *>(in + 4 * g); },
        [&](int64_t g, const uint2 &w) {
            const int32_t r[4] = {interpolatePair(pairs, int32_t(int16_t(w.x))), interpolatePair(pairs, int32_t(w.x) >> 16),
                                  interpolatePair(pairs, int32_t(int16_t(w.y))), interpolatePair(pairs, int32_t(w.y) >> 16)};
            store4<int32_t>(out + 4 * g, r);
        });
    GRID_STRIDE(g, rest) {
        out[4 * groups + g] = interpolatePair(pairs, in[4 * groups + g]);
    }
}

// ---- ADD / SUB / MUL on int32 (elementwise_binary.comp:146-173, mul.comp:24-59) ---------------------------------
// B_MODE: 0 = same shape, 1 = one value per row of `rowLen` elements (a multiple of 4), 2 = one value, 3 = one value per
// row of any length.
enum { kVecAdd = 0, kVecSub = 1, kVecMul = 2 };
template <int OP> __device__ __forceinline__ int32_t binaryI32(int32_t x, int32_t y, uint32_t shift) {
    if (OP == kVecAdd) {
        return int32_t(uint32_t(x) + uint32_t(y));
    }
    if (OP == kVecSub) {
        return int32_t(uint32_t(x) - uint32_t(y));
    }
    int64_t p = int64_t(x) * int64_t(y);
    if (shift > 0) {
        p = int64_t(uint64_t(p) + (1ull << ((shift - 1) & 63))) >> (shift & 63);
    }
    return int32_t(uint32_t(uint64_t(p)));
}

template <int OP, int B_MODE>
__global__ void binaryI32Kernel(const int32_t *__restrict__ a, const int32_t *__restrict__ b, int32_t *__restrict__ out,
                                int64_t groups, int rest, int rowLen, FastDiv divRow, uint32_t shift) {
    struct Operands {
        int4 x, y;
    };
    fourInFlight<Operands>(
        groups,
        [&](int64_t g) {
            Operands v;
            v.x = *reinterpret_cast<const int4 *>(a + 4 * g);
            if (B_MODE == 0) {
                v.y = *reinterpret_cast<const int4 *>(b + 4 * g);
            } else if (B_MODE == 3) {
                const uint32_t e = uint32_t(4 * g);
                v.y = make_int4(__ldg(b + fastDiv(e, divRow)), __ldg(b + fastDiv(e + 1, divRow)), __ldg(b + fastDiv(e + 2, divRow)),
                                __ldg(b + fastDiv(e + 3, divRow)));
            } else {
                const int32_t y = __ldg(b + (B_MODE == 1 ? (4 * g) / rowLen : 0));
                v.y = make_int4(y, y, y, y);
            }
            return v;
        },
        [&](int64_t g, const Operands &v) {
            *reinterpret_cast<int4 *>(out + 4 * g) = make_int4(binaryI32<OP>(v.x.x, v.y.x, shift), binaryI32<OP>(v.x.y, v.y.y, shift),
                                                               binaryI32<OP>(v.x.z, v.y.z, shift), binaryI32<OP>(v.x.w, v.y.w, shift));
        });
    GRID_STRIDE(g, rest) { // the last one to three elements, a thread each
        const int64_t e = 4 * groups + g;
        const int32_t y = B_MODE == 0 ? b[e] : (B_MODE == 2 ? b[0] : b[e / rowLen]);
        out[e] = binaryI32<OP>(a[e], y, shift);
    }
}

template <int OP>
void launchBinary(const int32_t *a, const int32_t *b, int32_t *out, int64_t n, int mode, int rowLen, uint32_t shift,
                  cudaStream_t s) {
    const int grid = gridFor(n / 4 + n % 4, kThreads, 16), rest = int(n % 4);
    const FastDiv divRow = makeFastDiv(rowLen);
    if (mode == 0) {
        binaryI32Kernel<OP, 0><<<grid, kThreads, 0, s>>>(a, b, out, n / 4, rest, rowLen, divRow, shift);
    } else if (mode == 1) {
        binaryI32Kernel<OP, 1><<<grid, kThreads, 0, s>>>(a, b, out, n / 4, rest, rowLen, divRow, shift);
    } else if (mode == 2) {
        binaryI32Kernel<OP, 2><<<grid, kThreads, 0, s>>>(a, b, out, n / 4, rest, rowLen, divRow, shift);
    } else {
        binaryI32Kernel<OP, 3><<<grid, kThreads, 0, s>>>(a, b, out, n / 4, rest, rowLen, divRow, shift);
    }
}

// ---- CLAMP on int8 (clamp.comp:24-53) -----------------------------------------------------------------------
// Four bytes at a time as even and odd bytes moved to the high byte of 16-bit lanes, whose signed order is the bytes'
// (byte by byte the extraction and packing took longer than the memory: 64 x 112 x 112 x 64 25.1 us, now 21.1).
__device__ __forceinline__ uint32_t clampBytes(uint32_t w, uint32_t lo, uint32_t hi) {
    const uint32_t even = __vmins2(__vmaxs2(__byte_perm(w, 0u, 0x2404), lo), hi), odd = __vmins2(__vmaxs2(w & 0xff00ff00u, lo), hi);
    return __byte_perm(even, odd, 0x7351);
}
__global__ void clampI8Kernel(const int8_t *__restrict__ in, int8_t *__restrict__ out, int64_t groups, int rest, int lo, int hi) {
    const uint32_t loLanes = (uint32_t(lo) & 0xffu) * 0x01000100u, hiLanes = (uint32_t(hi) & 0xffu) * 0x01000100u;
    fourInFlight<uint4>(
        groups, [&](int64_t g) { return *reinterpret_cast<const uint4 *>(in + 16 * g); },
        [&](int64_t g, const uint4 &w) {
            *reinterpret_cast<uint4 *>(out + 16 * g) = make_uint4(clampBytes(w.x, loLanes, hiLanes), clampBytes(w.y, loLanes, hiLanes),
                                                                  clampBytes(w.z, loLanes, hiLanes), clampBytes(w.w, loLanes, hiLanes));
        });
    GRID_STRIDE(g, rest) { // the last elements, a thread each
        const int64_t e = 16 * groups + g;
        out[e] = int8_t(min(max(int(in[e]), lo), hi));
    }
}

// ---- fused rows of a quantised softmax ---------------------------------------------------------------------------
// Element access of the two fused kernels below: 16-byte vectors where the tensors allow it, single elements where
// an application tensor sits at an odd address.
template <bool VEC> __device__ __forceinline__ void loadFourI32(const int32_t *p, int32_t (&v)[4]) {
    if (VEC) {
        load4<int32_t>(p, v);
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[k] = p[k];
        }
    }
}
template <bool VEC, typename T> __device__ __forceinline__ void storeFour(T *p, const int32_t (&v)[4]) {
    if (VEC) {
        store4<T>(p, v);
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            p[k] = T(v[k]);
        }
    }
}

// REDUCE_MAX(x) -> SUB(x, max) -> RESCALE (to int16) -> TABLE (int16 -> int32), and REDUCE_SUM of the TABLE's output
// (reduce.comp:24-70, elementwise_binary.comp:146-173, rescale.comp:27-72, table.comp): one warp per row, the row read
// twice (the second time from cache), every step with the arithmetic of the operator's own kernel above.
template <bool VEC>
__global__ void rowExpKernel(const int32_t *__restrict__ x, int32_t *__restrict__ e, int32_t *__restrict__ sums, int64_t rows,
                             int len, const int16_t *__restrict__ table, DevRescale r) {
    __shared__ int16_t lut[513];
    for (int i = threadIdx.x; i < 513; i += blockDim.x) {
        lut[i] = table[i];
    }
    __syncthreads();
    const FastRescale f = makeFastRescale(__ldg(r.mult), int32_t(__ldg(r.shift)), r.inZp, r.doubleRound != 0);
    const int lane = threadIdx.x & 31;
    const int64_t warp = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t warps = (int64_t(gridDim.x) * blockDim.x) >> 5;
    for (int64_t row = warp; row < rows; row += warps) {
        const int32_t *src = x + row * len;
        int32_t *dst = e + row * len;
        int32_t top = lowestOf<int32_t>();
        for (int i = lane * 4; i < len; i += 128) {
            int32_t v[4];
            loadFourI32<VEC>(src + i, v);
            top = max(max(top, v[0]), max(v[1], max(v[2], v[3])));
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            top = max(top, __shfl_xor_sync(0xffffffffu, top, d));
        }
        int32_t acc = 0;
        for (int i = lane * 4; i < len; i += 128) {
            int32_t v[4], out[4];
            loadFourI32<VEC>(src + i, v);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int32_t diff = int32_t(uint32_t(v[k]) - uint32_t(top));
                const int32_t q = fastRescale(f, diff, r.outZp, r.lo, r.hi); // an int16 value
                const int32_t index = (q + 32768) >> 7;
                const int32_t fraction = q & 0x7f;
                const int32_t base = lut[index], next = lut[index + 1];
                out[k] = int32_t((uint32_t(base) << 7) + uint32_t(next - base) * uint32_t(fraction));
                acc = int32_t(uint32_t(acc) + uint32_t(out[k]));
            }
            storeFour<VEC, int32_t>(dst + i, out);
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            acc = int32_t(uint32_t(acc) + uint32_t(__shfl_xor_sync(0xffffffffu, acc, d)));
        }
        if (lane == 0) {
            sums[row] = acc;
        }
    }
}

// MUL(a, b, shift) -> RESCALE [-> CLAMP] (mul.comp:24-59, rescale.comp:27-72).  B_MODE as in binaryI32Kernel.
template <typename OUT, int B_MODE, bool VEC>
__global__ void mulRescaleKernel(const int32_t *__restrict__ a, const int32_t *__restrict__ b, OUT *__restrict__ out,
                                 int64_t groups, int rowLen, uint32_t shift, DevRescale r) {
    const FastRescale f = makeFastRescale(__ldg(r.mult), int32_t(__ldg(r.shift)), r.inZp, r.doubleRound != 0);
    GRID_STRIDE(g, groups) {
        int32_t x[4], y[4], res[4];
        loadFourI32<VEC>(a + 4 * g, x);
        if (B_MODE == 0) {
            loadFourI32<VEC>(b + 4 * g, y);
        } else {
            const int32_t v = __ldg(b + (B_MODE == 1 ? (4 * g) / rowLen : 0));
            y[0] = y[1] = y[2] = y[3] = v;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            int64_t p = int64_t(x[k]) * int64_t(y[k]);
            if (shift > 0) {
                p = int64_t(uint64_t(p) + (1ull << ((shift - 1) & 63))) >> (shift & 63);
            }
            res[k] = fastRescale(f, int32_t(uint32_t(uint64_t(p))), r.outZp, r.lo, r.hi);
        }
        storeFour<VEC, OUT>(out + 4 * g, res);
    }
}

// ---- REDUCE_SUM / MAX / MIN along the last axis (reduce.comp:24-70) ------------------------------------------
// One warp per row: lanes stride through the row four elements at a time, then combine with shuffles.  Integer
// addition wraps, so the order of the partial sums does not change the result.
// VEC: rows start on four-element boundaries; otherwise a lane takes single elements, still coalesced.
template <typename T, int OP, bool VEC>
__global__ void rowReduceKernel(const T *__restrict__ in, T *__restrict__ out, int64_t rows, int len) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t warps = (int64_t(gridDim.x) * blockDim.x) >> 5;
    for (int64_t row = warp; row < rows; row += warps) {
        const T *src = in + row * len;
        int32_t acc = OP == RED_SUM ? 0 : (OP == RED_MAX ? lowestOf<T>() : highestOf<T>());
        const auto take = [&](int32_t v) {
            if (OP == RED_SUM) {
                acc = int32_t(uint32_t(acc) + uint32_t(v));
            } else if (OP == RED_MAX) {
                acc = max(acc, v);
            } else {
                acc = min(acc, v);
            }
        };
        if (VEC) {
            for (int i = lane * 4; i < len; i += 4 * 128) { // four loads at once
                int32_t v[4][4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (i + 128 * q < len) {
                        load4<T>(src + i + 128 * q, v[q]);
                    }
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (i + 128 * q < len) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            take(v[q][k]);
                        }
                    }
                }
            }
        } else {
#pragma unroll 4
            for (int i = lane; i < len; i += 32) {
                take(int32_t(__ldg(src + i)));
            }
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            const int32_t o = __shfl_xor_sync(0xffffffffu, acc, d);
            if (OP == RED_SUM) {
                acc = int32_t(uint32_t(acc) + uint32_t(o));
            } else if (OP == RED_MAX) {
                acc = max(acc, o);
            } else {
                acc = min(acc, o);
            }
        }
        if (lane == 0) {
            out[row] = T(acc); // a sum of T keeps T's low bits: the generic kernel wraps to the type after every step
        }
    }
}

template <typename T> void launchRowReduce(int32_t op, const TView &in, const TView &out, int64_t rows, int len, cudaStream_t s) {
    const int grid = gridFor(rows * 32, kThreads, 16);
    const T *pi = reinterpret_cast<const T *>(in.ptr);
    T *po = reinterpret_cast<T *>(out.ptr);
    const bool vec = aligned16(in.ptr) && len % 4 == 0;
    const auto launch = [&](auto vecKernel, auto kernel) { (vec ? vecKernel : kernel)<<<grid, kThreads, 0, s>>>(pi, po, rows, len); };
    if (op == RED_SUM) {
        launch(rowReduceKernel<T, RED_SUM, true>, rowReduceKernel<T, RED_SUM, false>);
    } else if (op == RED_MAX) {
        launch(rowReduceKernel<T, RED_MAX, true>, rowReduceKernel<T, RED_MAX, false>);
    } else {
        launch(rowReduceKernel<T, RED_MIN, true>, rowReduceKernel<T, RED_MIN, false>);
    }
}

// ---- TRANSPOSE that keeps the last axis (transpose.comp:19-32) -------------------------------------------------
// Rows of the last axis move as wholes: a thread copies 16 bytes; only the row index is permuted.  The index is
// taken apart with multiply-high divisions by constants made on the host (a 64-bit division per axis and thread was
// most of this kernel's time).
struct RowPermute {
    FastDiv outDims[kMaxRank];  // output dims without the last axis
    int64_t inStride[kMaxRank]; // input byte stride of the axis each output axis comes from
    FastDiv chunksPerRow;
    int rank;                   // number of outer axes
};

__global__ void transposeRowsKernel(const uint8_t *__restrict__ in, uint8_t *__restrict__ out, int64_t chunks, RowPermute p) {
    GRID_STRIDE(e, chunks) { // the launcher refuses 2^31 chunks and more
        uint32_t row = fastDiv(uint32_t(e), p.chunksPerRow);
        const uint32_t chunk = uint32_t(e) - row * p.chunksPerRow.d;
        int64_t src = 0;
#pragma unroll
        for (int i = kMaxRank - 1; i >= 0; --i) {
            if (i < p.rank) {
                const uint32_t q = fastDiv(row, p.outDims[i]);
                src += int64_t(row - q * p.outDims[i].d) * p.inStride[i];
                row = q;
            }
        }
        *reinterpret_cast<int4 *>(out + 16 * e) = __ldg(reinterpret_cast<const int4 *>(in + src + 16 * int64_t(chunk)));
    }
}

// ---- TRANSPOSE that swaps the last axis with another one, one-byte elements ------------------------------------
// out[..., c, r] = in[..., r (axis p), ..., c (last axis)]: per combination of the other axes a 2-D transpose of
// an R x Ccols byte matrix whose rows are `inRowStride` bytes apart.  No shared memory: a lane reads 8 rows x 16
// bytes (neighbouring lanes take the two halves of a 32-byte sector), transposes the eight 4 x 4 byte blocks in
// registers with byte permutes, and writes 16 double words, one to each of 16 output rows; the lanes of a warp
// that share a column half hold consecutive row octets, so every such store of the warp is two runs of 128
// contiguous bytes.
struct BatchPermute {
    FastDiv outDims[kMaxRank];  // output dims of the outer axes (all but the last two)
    int64_t inStride[kMaxRank]; // input byte stride of the axis each of them comes from
    FastDiv perBatch;           // warps per matrix
    FastDiv colGroups;          // 32-column groups per matrix
    int rank;
};

__global__ void __launch_bounds__(256) transposeLast2BytesKernel(const uint8_t *__restrict__ in, uint8_t *__restrict__ out,
                                                                 int R, int Ccols, int64_t inRowStride, int64_t warps,
                                                                 BatchPermute p) {
    const int lane = threadIdx.x & 31;
    for (int64_t wid = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; wid < warps;
         wid += (int64_t(gridDim.x) * blockDim.x) >> 5) {
        uint32_t batch = fastDiv(uint32_t(wid), p.perBatch);
        const uint32_t inMat = uint32_t(wid) - batch * p.perBatch.d;
        const uint32_t rowGroup = fastDiv(inMat, p.colGroups);
        const int c0 = int(inMat - rowGroup * p.colGroups.d) * 32 + (lane & 1) * 16;
        const int r = (int(rowGroup) * 16 + (lane >> 1)) * 8;
        uint8_t *dst = out + int64_t(batch) * R * Ccols;
        int64_t src = 0;
#pragma unroll
        for (int i = kMaxRank - 1; i >= 0; --i) {
            if (i < p.rank) {
                const uint32_t q = fastDiv(batch, p.outDims[i]);
                src += int64_t(batch - q * p.outDims[i].d) * p.inStride[i];
                batch = q;
            }
        }
        if (r >= R || c0 >= Ccols) { // R is a multiple of 8 and Ccols of 16: a block is inside or outside as a whole
            continue;
        }
        uint32_t w[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int4 v = __ldg(reinterpret_cast<const int4 *>(in + src + int64_t(r + i) * inRowStride + c0));
            w[i][0] = uint32_t(v.x), w[i][1] = uint32_t(v.y), w[i][2] = uint32_t(v.z), w[i][3] = uint32_t(v.w);
        }
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            // rows r .. r+7, columns c0 + 4g .. +3  ->  output rows c0 + 4g + k, bytes r .. r+7
            uint32_t lo[4], hi[4];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t t0 = __byte_perm(w[4 * h][g], w[4 * h + 1][g], 0x5140);
                const uint32_t t1 = __byte_perm(w[4 * h + 2][g], w[4 * h + 3][g], 0x5140);
                const uint32_t t2 = __byte_perm(w[4 * h][g], w[4 * h + 1][g], 0x7362);
                const uint32_t t3 = __byte_perm(w[4 * h + 2][g], w[4 * h + 3][g], 0x7362);
                uint32_t *o = h == 0 ? lo : hi;
                o[0] = __byte_perm(t0, t1, 0x5410), o[1] = __byte_perm(t0, t1, 0x7632);
                o[2] = __byte_perm(t2, t3, 0x5410), o[3] = __byte_perm(t2, t3, 0x7632);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                *reinterpret_cast<uint2 *>(dst + int64_t(c0 + 4 * g + k) * R + r) = make_uint2(lo[k], hi[k]);
            }
        }
    }
}

} // namespace

bool vecRescale(const TView &in, const TView &out, const TView &mult, const TView &shift, const RescaleAttr &a, cudaStream_t s,
                int *rc) {
    const int64_t n = packedNumel(in);
    if (n <= 0 || n != packedNumel(out) || !sameShape(in, out) || !signedInt(in.dtype) || !signedInt(out.dtype) ||
        !aligned16(in.ptr) || !aligned16(out.ptr) || mult.dtype != MLEL_I32 || shift.dtype != MLEL_I8 ||
        packedNumel(mult) < 1 || packedNumel(shift) < 1 || n >= (int64_t(1) << 40)) {
        return false;
    }
    const int64_t C = out.dims[out.rank - 1];
    if (a.perChannel && (C < 4 || packedNumel(mult) != C || packedNumel(shift) != C)) {
        return false;
    }
#define MLEL_RESCALE_CASE(IN_ID, IN_T, OUT_ID, OUT_T)                                                                          \
    if (in.dtype == IN_ID && out.dtype == OUT_ID) {                                                                            \
        launchRescale<IN_T, OUT_T>(in, out, mult, shift, a, n, s);                                                             \
        *rc = finish("RESCALE");                                                                                               \
        return true;                                                                                                           \
    }
    MLEL_RESCALE_CASE(MLEL_I32, int32_t, MLEL_I8, int8_t)
    MLEL_RESCALE_CASE(MLEL_I32, int32_t, MLEL_I16, int16_t)
    MLEL_RESCALE_CASE(MLEL_I32, int32_t, MLEL_I32, int32_t)
    MLEL_RESCALE_CASE(MLEL_I8, int8_t, MLEL_I32, int32_t)
    MLEL_RESCALE_CASE(MLEL_I8, int8_t, MLEL_I8, int8_t)
    MLEL_RESCALE_CASE(MLEL_I16, int16_t, MLEL_I32, int32_t)
    MLEL_RESCALE_CASE(MLEL_I16, int16_t, MLEL_I16, int16_t)
    MLEL_RESCALE_CASE(MLEL_I16, int16_t, MLEL_I8, int8_t)
    MLEL_RESCALE_CASE(MLEL_I8, int8_t, MLEL_I16, int16_t)
#undef MLEL_RESCALE_CASE
    return false;
}

bool vecTable(const TView &in, const TView &out, const TView &table, cudaStream_t s, int *rc) {
    const int64_t n = packedNumel(in);
    if (n <= 0 || n != packedNumel(out) || !sameShape(in, out) || !aligned16(in.ptr) || !aligned16(out.ptr) ||
        packedNumel(table) < 0) {
        return false;
    }
    if (in.dtype == MLEL_I8 && out.dtype == MLEL_I8 && table.dtype == MLEL_I8 && packedNumel(table) == 256) {
        if (n >= int64_t(1) << 23) {
            tableI8LanesKernel<<<gridFor(n / 16 + n % 16, kLaneTableThreads, 2), kLaneTableThreads, 0, s>>>(
                reinterpret_cast<const int8_t *>(in.ptr), reinterpret_cast<int8_t *>(out.ptr), n / 16, int(n % 16),
                reinterpret_cast<const int8_t *>(table.ptr));
            *rc = finish("TABLE");
            return true;
        }
        // (the GELU between two projections: its blocks are scheduled while the product before it drains)
        launchOverlapped(tableI8Kernel, gridFor(n / 16 + n % 16, kThreads, 16), kThreads, 0, s,
                         reinterpret_cast<const int8_t *>(in.ptr), reinterpret_cast<int8_t *>(out.ptr), n / 16, int(n % 16),
                         reinterpret_cast<const int8_t *>(table.ptr));
        *rc = finish("TABLE");
        return true;
    }
    if (in.dtype == MLEL_I16 && out.dtype == MLEL_I32 && table.dtype == MLEL_I16 && packedNumel(table) == 513) {
        tableI16Kernel<<<gridFor(n / 4 + n % 4, kThreads, 16), kThreads, 0, s>>>(reinterpret_cast<const int16_t *>(in.ptr),
                                                                        reinterpret_cast<int32_t *>(out.ptr), n / 4, int(n % 4),
                                                                        reinterpret_cast<const int16_t *>(table.ptr));
        *rc = finish("TABLE");
        return true;
    }
    return false;
}

// op: BIN_ADD or BIN_SUB of ops.hpp, or -1 for MUL with `shift`.
bool vecBinaryI32(int32_t op, const TView &a, const TView &b, const TView &out, uint32_t shift, cudaStream_t s, int *rc) {
    const int64_t n = packedNumel(out);
    if (n <= 0 || a.dtype != MLEL_I32 || b.dtype != MLEL_I32 || out.dtype != MLEL_I32 || packedNumel(a) != n ||
        !sameShape(a, out) || packedNumel(b) < 1 || !aligned16(a.ptr) || !aligned16(out.ptr) || shift > 62) {
        return false;
    }
    const int rowLen = int(out.dims[out.rank - 1]);
    int mode;
    if (sameShape(b, out)) {
        mode = 0;
        if (!aligned16(b.ptr)) {
            return false;
        }
    } else if (packedNumel(b) == 1 && b.rank == out.rank) {
        mode = 2;
    } else if (rowBroadcast(b, out) && (rowLen % 4 == 0 || n < (int64_t(1) << 31))) {
        mode = rowLen % 4 == 0 ? 1 : 3;
    } else {
        return false;
    }
    const auto *pa = reinterpret_cast<const int32_t *>(a.ptr), *pb = reinterpret_cast<const int32_t *>(b.ptr);
    auto *po = reinterpret_cast<int32_t *>(out.ptr);
    if (op == BIN_ADD) {
        launchBinary<kVecAdd>(pa, pb, po, n, mode, rowLen, 0, s);
    } else if (op == BIN_SUB) {
        launchBinary<kVecSub>(pa, pb, po, n, mode, rowLen, 0, s);
    } else if (op == -1) {
        launchBinary<kVecMul>(pa, pb, po, n, mode, rowLen, shift, s);
    } else {
        return false;
    }
    *rc = finish("element-wise int32");
    return true;
}

bool vecClampI8(const TView &in, const TView &out, int64_t lo, int64_t hi, cudaStream_t s, int *rc) {
    const int64_t n = packedNumel(in);
    if (n <= 0 || n != packedNumel(out) || !sameShape(in, out) || in.dtype != MLEL_I8 || out.dtype != MLEL_I8 ||
        !aligned16(in.ptr) || !aligned16(out.ptr)) {
        return false;
    }
    clampI8Kernel<<<gridFor(n / 16 + n % 16, kThreads, 16), kThreads, 0, s>>>(
        reinterpret_cast<const int8_t *>(in.ptr), reinterpret_cast<int8_t *>(out.ptr), n / 16, int(n % 16), int(lo), int(hi));
    *rc = finish("CLAMP");
    return true;
}

bool vecRowReduce(int32_t op, const TView &in, const TView &out, uint32_t axis, cudaStream_t s, int *rc) {
    const int64_t n = packedNumel(in), rows = packedNumel(out);
    if (n <= 0 || rows <= 0 || in.rank < 1 || int(axis) != in.rank - 1 || out.rank != in.rank || out.dims[axis] != 1 ||
        in.dtype != out.dtype || !signedInt(in.dtype) || (op != RED_SUM && op != RED_MAX && op != RED_MIN)) {
        return false;
    }
    const int64_t len = in.dims[axis];
    if (len > (1 << 30) || rows * len != n) {
        return false;
    }
    if (in.dtype == MLEL_I32) {
        launchRowReduce<int32_t>(op, in, out, rows, int(len), s);
    } else if (in.dtype == MLEL_I16) {
        launchRowReduce<int16_t>(op, in, out, rows, int(len), s);
    } else {
        launchRowReduce<int8_t>(op, in, out, rows, int(len), s);
    }
    *rc = finish("REDUCE");
    return true;
}

bool vecTransposeRows(const TView &in, const TView &out, const uint32_t *perms, cudaStream_t s, int *rc) {
    const int64_t n = packedNumel(in);
    const int rank = out.rank;
    if (n <= 0 || n != packedNumel(out) || rank < 2 || in.rank != rank || in.dtype != out.dtype ||
        int(perms[rank - 1]) != rank - 1 || !aligned16(in.ptr) || !aligned16(out.ptr)) {
        return false;
    }
    const int64_t rowBytes = int64_t(out.dims[rank - 1]) * dtypeSize(out.dtype);
    if (rowBytes % 16 != 0 || rowBytes / 16 > (1 << 24)) {
        return false;
    }
    const int64_t chunks = n * dtypeSize(out.dtype) / 16;
    if (chunks >= (int64_t(1) << 31)) {
        return false;
    }
    RowPermute p{};
    p.rank = rank - 1;
    p.chunksPerRow = makeFastDiv(rowBytes / 16);
    for (int i = 0; i < rank - 1; ++i) {
        if (perms[i] >= uint32_t(rank - 1) || in.dims[perms[i]] != out.dims[i]) {
            return false;
        }
        p.outDims[i] = makeFastDiv(out.dims[i]);
        p.inStride[i] = in.strides[perms[i]];
    }
    transposeRowsKernel<<<gridFor(chunks, kThreads, 16), kThreads, 0, s>>>(reinterpret_cast<const uint8_t *>(in.ptr),
                                                                          reinterpret_cast<uint8_t *>(out.ptr), chunks, p);
    *rc = finish("TRANSPOSE");
    return true;
}

bool vecTransposeLast2Bytes(const TView &in, const TView &out, const uint32_t *perms, cudaStream_t s, int *rc) {
    const int64_t n = packedNumel(in);
    const int rank = out.rank;
    if (n <= 0 || n != packedNumel(out) || rank < 2 || in.rank != rank || in.dtype != out.dtype || dtypeSize(out.dtype) != 1 ||
        int(perms[rank - 2]) != rank - 1 || int(perms[rank - 1]) == rank - 1 || !aligned16(in.ptr) || !aligned16(out.ptr)) {
        return false;
    }
    const uint32_t pAxis = perms[rank - 1];
    const int64_t R = in.dims[pAxis], Ccols = in.dims[rank - 1];
    const int64_t inRowStride = in.strides[pAxis];
    if (R % 8 != 0 || Ccols % 16 != 0 || inRowStride % 16 != 0 || out.dims[rank - 1] != R || out.dims[rank - 2] != Ccols) {
        return false;
    }
    BatchPermute p{};
    p.rank = rank - 2;
    int64_t batches = 1;
    for (int i = 0; i < rank - 2; ++i) {
        if (perms[i] >= uint32_t(rank) || perms[i] == pAxis || int(perms[i]) == rank - 1 || in.dims[perms[i]] != out.dims[i]) {
            return false;
        }
        p.outDims[i] = makeFastDiv(out.dims[i]);
        p.inStride[i] = in.strides[perms[i]];
        if (p.inStride[i] % 16 != 0) {
            return false;
        }
        batches *= out.dims[i];
    }
    const int64_t colGroups = (Ccols + 31) / 32, rowGroups = (R + 127) / 128;
    const int64_t warps = batches * colGroups * rowGroups;
    if (warps >= (int64_t(1) << 31)) {
        return false;
    }
    p.perBatch = makeFastDiv(colGroups * rowGroups);
    p.colGroups = makeFastDiv(colGroups);
    transposeLast2BytesKernel<<<gridFor(warps * 32, 256, 8), 256, 0, s>>>(reinterpret_cast<const uint8_t *>(in.ptr),
                                                                        reinterpret_cast<uint8_t *>(out.ptr), int(R),
                                                                        int(Ccols), inRowStride, warps, p);
    *rc = finish("TRANSPOSE");
    return true;
}

namespace {

// out[row][first[g] + j] = staging[g][row][j] for j < count[g]: joins the column blocks that an all-gather left
// one after another (every block padded to `pitch` bytes per row) into rows of `total` bytes.  One thread moves
// 16 bytes when every block starts and ends on a 16-byte boundary (VEC = 16), else one byte.
struct ColumnBlocks {
    int32_t first[kMaxColumnBlocks];
    int32_t count[kMaxColumnBlocks];
};

template <int VEC>
__global__ void interleaveColumnsKernel(const uint8_t *__restrict__ staging, uint8_t *__restrict__ out, int64_t rows,
                                        int32_t blocks, int32_t pitch, int32_t total, ColumnBlocks cb) {
    const int64_t unitsPerRow = total / VEC;
    GRID_STRIDE(e, rows * unitsPerRow) {
        const int64_t row = e / unitsPerRow;
        const int32_t col = int32_t(e - row * unitsPerRow) * VEC;
        int g = 0;
        while (g + 1 < blocks && col >= cb.first[g + 1]) {
            ++g;
        }
        const uint8_t *src = staging + (int64_t(g) * rows + row) * pitch + (col - cb.first[g]);
        uint8_t *dst = out + row * int64_t(total) + col;
        if (VEC == 16) {
            *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(src);
        } else {
            *dst = *src;
        }
    }
}

} // namespace

int interleaveColumns(const void *staging, void *out, int64_t rows, int32_t blocks, int32_t pitch, const int32_t *first,
                      const int32_t *count, cudaStream_t s) {
    if (blocks < 1 || blocks > kMaxColumnBlocks || rows < 0 || pitch < 0) {
        setLastError("interleave columns: bad block description");
        return MLEL_ERROR_UNKNOWN;
    }
    ColumnBlocks cb{};
    int64_t total = 0;
    bool vec = (reinterpret_cast<uintptr_t>(staging) & 15u) == 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0 &&
               pitch % 16 == 0;
    for (int g = 0; g < blocks; ++g) {
        if (first[g] != total || count[g] < 0 || count[g] > pitch) {
            setLastError("interleave columns: blocks must follow one another and fit the pitch");
            return MLEL_ERROR_UNKNOWN;
        }
        cb.first[g] = first[g], cb.count[g] = count[g];
        total += count[g];
        vec = vec && first[g] % 16 == 0 && count[g] % 16 == 0;
    }
    if (total == 0 || rows == 0) {
        return MLEL_SUCCESS;
    }
    if (total >= (int64_t(1) << 31)) {
        setLastError("interleave columns: rows too long");
        return MLEL_ERROR_UNKNOWN;
    }
    const int64_t units = rows * (total / (vec ? 16 : 1));
    const int grid = int(std::min<int64_t>((units + 255) / 256, int64_t(kNumSMs) * 16));
    if (vec) {
        interleaveColumnsKernel<16><<<grid, 256, 0, s>>>(static_cast<const uint8_t *>(staging), static_cast<uint8_t *>(out),
                                                         rows, blocks, pitch, int32_t(total), cb);
    } else {
        interleaveColumnsKernel<1><<<grid, 256, 0, s>>>(static_cast<const uint8_t *>(staging), static_cast<uint8_t *>(out),
                                                        rows, blocks, pitch, int32_t(total), cb);
    }
    return finish("interleave columns");
}


int rowExpFused(const TView &x, const TView &table, const TView &e, const TView &sums, const DevRescale &r, cudaStream_t s) {
    const int len = int(x.dims[x.rank - 1]);
    const int64_t n = packedNumel(x);
    if (n <= 0 || len <= 0 || len % 4 != 0 || packedNumel(e) != n || packedNumel(sums) != n / len || packedNumel(table) != 513) {
        setLastError("fused softmax rows: operands do not match");
        return MLEL_ERROR_UNKNOWN;
    }
    const int64_t rows = n / len;
    const int grid = gridFor(rows * 32, kThreads, 16);
    const auto *px = reinterpret_cast<const int32_t *>(x.ptr);
    auto *pe = reinterpret_cast<int32_t *>(e.ptr);
    auto *ps = reinterpret_cast<int32_t *>(sums.ptr);
    const auto *pt = reinterpret_cast<const int16_t *>(table.ptr);
    if (aligned16(x.ptr) && aligned16(e.ptr)) {
        rowExpKernel<true><<<grid, kThreads, 0, s>>>(px, pe, ps, rows, len, pt, r);
    } else {
        rowExpKernel<false><<<grid, kThreads, 0, s>>>(px, pe, ps, rows, len, pt, r);
    }
    return finish("REDUCE_MAX+SUB+RESCALE+TABLE+REDUCE_SUM");
}

namespace {
template <typename OUT>
void launchMulRescale(const TView &a, const TView &b, const TView &out, int64_t n, int mode, int rowLen, uint32_t shift,
                      const DevRescale &r, cudaStream_t s) {
    const int grid = gridFor(n / 4, kThreads, 16);
    const auto *pa = reinterpret_cast<const int32_t *>(a.ptr);
    const auto *pb = reinterpret_cast<const int32_t *>(b.ptr);
    auto *po = reinterpret_cast<OUT *>(out.ptr);
    const bool vec = aligned16(a.ptr) && (mode != 0 || aligned16(b.ptr)) &&
                     (reinterpret_cast<uintptr_t>(out.ptr) & (4 * sizeof(OUT) - 1)) == 0;
#define MLEL_MUL_RESCALE(MODE)                                                                                     \
    if (vec) {                                                                                                     \
        mulRescaleKernel<OUT, MODE, true><<<grid, kThreads, 0, s>>>(pa, pb, po, n / 4, rowLen, shift, r);         \
    } else {                                                                                                       \
        mulRescaleKernel<OUT, MODE, false><<<grid, kThreads, 0, s>>>(pa, pb, po, n / 4, rowLen, shift, r);        \
    }
    if (mode == 0) {
        MLEL_MUL_RESCALE(0)
    } else if (mode == 1) {
        MLEL_MUL_RESCALE(1)
    } else {
        MLEL_MUL_RESCALE(2)
    }
#undef MLEL_MUL_RESCALE
}
} // namespace

int mulRescaleFused(const TView &a, const TView &b, const TView &out, uint32_t shift, const DevRescale &r, cudaStream_t s) {
    const int64_t n = packedNumel(a), nb = packedNumel(b);
    const int rowLen = int(a.dims[a.rank - 1]);
    if (n <= 0 || n % 4 != 0 || rowLen % 4 != 0 || packedNumel(out) != n || nb <= 0) {
        setLastError("fused MUL+RESCALE: operands do not match");
        return MLEL_ERROR_UNKNOWN;
    }
    const int mode = nb == n ? 0 : (nb == 1 ? 2 : 1);
    if (mode == 1 && nb != n / rowLen) {
        setLastError("fused MUL+RESCALE: second operand is neither per row nor a single value");
        return MLEL_ERROR_UNKNOWN;
    }
    if (out.dtype == MLEL_I8) {
        launchMulRescale<int8_t>(a, b, out, n, mode, rowLen, shift, r, s);
    } else if (out.dtype == MLEL_I16) {
        launchMulRescale<int16_t>(a, b, out, n, mode, rowLen, shift, r, s);
    } else {
        setLastError("fused MUL+RESCALE: output type");
        return MLEL_ERROR_UNKNOWN;
    }
    return finish("MUL+RESCALE");
}

} // namespace mlel
