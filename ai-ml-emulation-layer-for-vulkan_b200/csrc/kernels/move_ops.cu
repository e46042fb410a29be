// Data movement on strided tensors as copies of contiguous runs, and the index operators whose runs are whole
// channel rows: TRANSPOSE, CONCAT, SLICE, TILE, REVERSE, RESIZE (NEAREST) and ARGMAX along the last axis.
//
// What bounds these is memory, but only once the index arithmetic is out of the way: one thread per element with an
// unravel of up to six 32-bit divisions on either side moved 46 elements per nanosecond whatever the element size (a
// CONCAT of 4.7 MB of int8 took 102 us).  Here every move is reduced on the host to
//   dst[dstBase + sum i_k * dstStride_k + r] = src[srcBase + sum i_k * srcStride_k + r],   r < run,
// adjacent axes that both sides walk alike are merged (a CONCAT along the channels has one outer axis, a SLICE of
// rows none), and a thread moves the widest unit (16 to 1 bytes) that divides the run, all strides and both addresses,
// with multiply-high divisions.  Measured on a B200 (events around single launches, about 6 us of which are the launch):
// CONCAT of two 4.7 MB int8 tensors 205 -> 8.2 us, RESIZE of 8.3 MB 96 -> 9.0 us, SLICE of 4.1 MB 92 -> 6.3 us.
#include <algorithm>
#include <string>

#include "device_common.cuh"
#include "gemm_i8_tcgen05.hpp"
#include "kernels.hpp"
#include "nearest_source.hpp"
#include "launch_overlapped.cuh"

namespace mlel {

namespace {

constexpr int kMaxMoveAxes = 6;
constexpr int kMaxMoveParts = 4;

int finish(const char *what) {
    const cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) {
        setLastError(std::string(what) + ": " + cudaGetErrorString(err));
        return MLEL_ERROR_DEVICE;
    }
    return MLEL_SUCCESS;
}

// One strided copy: `axes` outer axes (the last varies fastest) over runs of contiguous bytes.
struct RunMove {
    const uint8_t *src;
    uint8_t *dst;
    uint32_t units; // units of the whole copy
    int32_t axes;
    FastDiv unitsPerRun;
    FastDiv dims[kMaxMoveAxes];
    int64_t srcStride[kMaxMoveAxes], dstStride[kMaxMoveAxes];
};
struct RunMoves {
    RunMove part[kMaxMoveParts];
};

// Four units per thread and step, all loads before the first store; blockIdx.y selects the part.
template <typename UNIT> __global__ void __launch_bounds__(256) runMoveKernel(const __grid_constant__ RunMoves moves) {
    dependencySync();
    const RunMove &m = moves.part[blockIdx.y];
    const uint32_t step = gridDim.x * blockDim.x;
    for (uint64_t first = blockIdx.x * blockDim.x + threadIdx.x; first < m.units; first += uint64_t(step) * 4) {
        UNIT v[4];
        int64_t dst[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint64_t e = first + uint64_t(u) * step;
            dst[u] = -1;
            if (e < m.units) {
                uint32_t row = fastDiv(uint32_t(e), m.unitsPerRun);
                const int64_t r = int64_t(uint32_t(e) - row * m.unitsPerRun.d) * int64_t(sizeof(UNIT));
                int64_t so = r, to = r;
                for (int k = m.axes - 1; k >= 0; --k) {
                    const uint32_t q = k > 0 ? fastDiv(row, m.dims[k]) : 0u;
                    const int64_t i = row - q * m.dims[k].d;
                    so += i * m.srcStride[k];
                    to += i * m.dstStride[k];
                    row = q;
                }
                v[u] = *reinterpret_cast<const UNIT *>(m.src + so);
                dst[u] = to;
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (dst[u] >= 0) {
                *reinterpret_cast<UNIT *>(m.dst + dst[u]) = v[u];
            }
        }
    }
}

// Description of one copy before it is reduced: every axis of the element grid with its byte strides.
struct MoveAxes {
    int n = 0;
    int64_t dim[2 * kMaxRank], src[2 * kMaxRank], dst[2 * kMaxRank];
    void add(int64_t d, int64_t s, int64_t t) {
        if (d != 1) {
            dim[n] = d, src[n] = s, dst[n] = t;
            ++n;
        }
    }
};

// Reduces `a` (elements of `elem` bytes) to runs; false when it does not fit a RunMove.  *unit is narrowed to the
// widest access this copy allows.
bool makeRunMove(MoveAxes a, int64_t elem, const char *src, char *dst, RunMove *m, int64_t *run, int64_t *unit) {
    *run = elem;
    while (a.n > 0 && a.src[a.n - 1] == *run && a.dst[a.n - 1] == *run) {
        *run *= a.dim[a.n - 1];
        --a.n;
    }
    // merge an axis into the one inside it where both sides step over exactly that axis
    int out = 0;
    MoveAxes merged;
    for (int k = a.n - 1; k >= 0; --k) { // collected inside out
        if (out > 0 && a.src[k] == merged.src[out - 1] * merged.dim[out - 1] &&
            a.dst[k] == merged.dst[out - 1] * merged.dim[out - 1]) {
            merged.dim[out - 1] *= a.dim[k];
        } else {
            merged.dim[out] = a.dim[k], merged.src[out] = a.src[k], merged.dst[out] = a.dst[k];
            ++out;
        }
    }
    if (out > kMaxMoveAxes) {
        return false;
    }
    uint64_t bits = uint64_t(*run) | reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst);
    m->axes = out;
    for (int k = 0; k < out; ++k) {
        const int j = out - 1 - k;
        m->dims[k] = makeFastDiv(merged.dim[j]);
        m->srcStride[k] = merged.src[j];
        m->dstStride[k] = merged.dst[j];
        bits |= uint64_t(merged.src[j]) | uint64_t(merged.dst[j]);
        if (merged.dim[j] <= 0 || merged.dim[j] >= (int64_t(1) << 31)) {
            return false;
        }
    }
    while ((bits & uint64_t(*unit - 1)) != 0) {
        *unit >>= 1;
    }
    m->src = reinterpret_cast<const uint8_t *>(src);
    m->dst = reinterpret_cast<uint8_t *>(dst);
    return true;
}

int64_t numelOf(const TView &t) {
    int64_t n = 1;
    for (int i = 0; i < t.rank; ++i) {
        n *= t.dims[i];
    }
    return n;
}

// Launches up to kMaxMoveParts copies of one destination tensor as one kernel; false: nothing was launched.
bool launchRunMoves(RunMove *parts, const int64_t *runs, const int64_t *bytes, int count, int64_t unit, const char *what,
                    cudaStream_t s, int *rc) {
    RunMoves moves{};
    int64_t most = 0;
    for (int k = 0; k < count; ++k) {
        const int64_t units = bytes[k] / unit;
        if (units >= (int64_t(1) << 31) || runs[k] / unit >= (int64_t(1) << 31)) {
            return false;
        }
        parts[k].units = uint32_t(units);
        parts[k].unitsPerRun = makeFastDiv(runs[k] / unit);
        moves.part[k] = parts[k];
        most = std::max(most, units);
    }
    // enough blocks for every SM to hold eight; a thread's four units come first, so small copies stay one wave
    const dim3 grid(unsigned(gridFor((most + 3) / 4, kThreads, 16)), unsigned(count));
    switch (unit) {
    case 16:
        launchOverlapped(runMoveKernel<uint4>, dim3(grid), kThreads, 0, s, moves);
        break;
    case 8:
        launchOverlapped(runMoveKernel<uint2>, dim3(grid), kThreads, 0, s, moves);
        break;
    case 4:
        launchOverlapped(runMoveKernel<uint32_t>, dim3(grid), kThreads, 0, s, moves);
        break;
    case 2:
        launchOverlapped(runMoveKernel<uint16_t>, dim3(grid), kThreads, 0, s, moves);
        break;
    default:
        launchOverlapped(runMoveKernel<uint8_t>, dim3(grid), kThreads, 0, s, moves);
        break;
    }
    *rc = finish(what);
    return true;
}

bool moveOne(const MoveAxes &a, int64_t elem, const char *src, char *dst, int64_t numel, const char *what, cudaStream_t s,
             int *rc) {
    RunMove m{};
    int64_t run = 0, unit = 16;
    const int64_t bytes = numel * elem;
    return numel > 0 && makeRunMove(a, elem, src, dst, &m, &run, &unit) &&
           launchRunMoves(&m, &run, &bytes, 1, unit, what, s, rc);
}

bool sameElement(const TView &in, const TView &out) {
    return in.rank == out.rank && dtypeSize(in.dtype) == dtypeSize(out.dtype) && dtypeSize(in.dtype) > 0;
}

// ---- TRANSPOSE that moves another axis to the last place (transpose.comp:19-32) --------------------------------
// Per combination of the other axes a 2-D transpose of R rows (contiguous in the output) by C columns (contiguous in
// the input): 64 x 64 tiles through shared memory, reads and writes both along contiguous elements.  The tile's rows are
// an odd number of words apart, so that a warp's column reads fall into 32 banks.  (Whole multiples of 8 x 16 one-byte
// elements have a kernel without shared memory, vecTransposeLast2Bytes.)  36 matrices of 197 x 64 bytes: 14.2 -> 7.2 us.
struct TileTranspose {
    FastDiv tilesC, tilesPerMatrix;
    FastDiv dims[kMaxRank];
    int64_t srcStride[kMaxRank], dstStride[kMaxRank];
    int32_t axes, R, C;
    int64_t srcRow, dstRow; // byte strides of R in the input and of C in the output
};

template <typename T>
__global__ void __launch_bounds__(256) tileTransposeKernel(const uint8_t *in, uint8_t *out,
                                                           uint32_t tiles, const __grid_constant__ TileTranspose p) {
    dependencySync();
    constexpr int kPitch = 64 * int(sizeof(T)) + 4;
    __shared__ __align__(16) uint8_t tile[64 * kPitch];
    const int x = threadIdx.x & 63, y0 = threadIdx.x >> 6;
    for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        uint32_t matrix = fastDiv(t, p.tilesPerMatrix);
        const uint32_t inMatrix = t - matrix * p.tilesPerMatrix.d;
        const uint32_t tr = fastDiv(inMatrix, p.tilesC);
        const int r0 = int(tr) * 64, c0 = int(inMatrix - tr * p.tilesC.d) * 64;
        int64_t so = 0, to = 0;
        for (int k = p.axes - 1; k >= 0; --k) {
            const uint32_t q = fastDiv(matrix, p.dims[k]);
            const int64_t i = matrix - q * p.dims[k].d;
            so += i * p.srcStride[k];
            to += i * p.dstStride[k];
            matrix = q;
        }
        T v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int r = r0 + y0 + 4 * i, c = c0 + x;
            v[i] = r < p.R && c < p.C ? *(reinterpret_cast<const T *>(in + so + int64_t(r) * p.srcRow) + c) : T(0);
        }
        __syncthreads(); // the previous tile has been read
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            *reinterpret_cast<T *>(&tile[(y0 + 4 * i) * kPitch + x * int(sizeof(T))]) = v[i];
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int c = c0 + y0 + 4 * i, r = r0 + x;
            if (r < p.R && c < p.C) {
                *(reinterpret_cast<T *>(out + to + int64_t(c) * p.dstRow) + r) =
                    *reinterpret_cast<const T *>(&tile[x * kPitch + (y0 + 4 * i) * int(sizeof(T))]);
            }
        }
    }
}

// ---- RESIZE, NEAREST (resize.comp:43-134): one source pixel per output pixel, its channels moved as units ---------
template <typename UNIT>
__global__ void __launch_bounds__(256)
    resizeNearestKernel(const uint8_t *in, uint8_t *out, uint32_t units, FastDiv perPixel, FastDiv divOW,
                        FastDiv divOH, uint32_t H, uint32_t W, ResizeAttr a) {
    dependencySync();
    const uint32_t step = gridDim.x * blockDim.x;
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < units; e += step) {
        const uint32_t pixel = fastDiv(e, perPixel), u = e - pixel * perPixel.d;
        const uint32_t line = fastDiv(pixel, divOW), ox = pixel - line * divOW.d;
        const uint32_t n = fastDiv(line, divOH), oy = line - n * divOH.d;
        const uint32_t y = nearestSource(oy, a.scale[0], a.scale[1], a.offset[0], H);
        const uint32_t x = nearestSource(ox, a.scale[2], a.scale[3], a.offset[1], W);
        UNIT v{}; // a position outside the image reads zero
        if (y < H && x < W) {
            v = reinterpret_cast<const UNIT *>(in)[(int64_t(n) * H + y) * W * perPixel.d + int64_t(x) * perPixel.d + u];
        }
        reinterpret_cast<UNIT *>(out)[e] = v;
        if (units - e <= step) {
            break; // e + step could wrap
        }
    }
}

// ---- CONCAT along the channels of tensors that are enlarged on the way (OP_FUSED_CONCAT) -----------------------------
// The joined tensor is written once and its sources are read where they lie; as RESIZE, SLICE and CONCAT the enlarged tensor went
// to memory and back twice (270 x 480, 64 channels of 135 x 240 beside 32: three launches of 2.5 to 4.7 us).  Where a pixel comes
// from is a table of rows and one of columns, made by the host: the shader's divisions per unit were most of RESIZE's time.
struct ConcatPart {
    const uint8_t *src;
    const int32_t *rows, *columns; // or null: the pixel itself
    uint32_t begin, units;         // units of a pixel of the result, first and count
    uint32_t H, W;
};
struct ConcatParts {
    ConcatPart part[kMaxResizedConcatInputs];
    uint32_t units; // of the result
    FastDiv perPixel, divOW, divOH;
};

template <typename UNIT>
__global__ void __launch_bounds__(256) concatResizedKernel(uint8_t *out, const __grid_constant__ ConcatParts p) {
    dependencySync();
    const uint32_t step = gridDim.x * blockDim.x;
    for (uint64_t first = blockIdx.x * blockDim.x + threadIdx.x; first < p.units; first += uint64_t(step) * 4) {
        UNIT v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint64_t at = first + uint64_t(j) * step;
            v[j] = UNIT{};
            if (at < p.units) {
                const uint32_t e = uint32_t(at), pixel = fastDiv(e, p.perPixel), u = e - pixel * p.perPixel.d;
                const uint8_t *src = p.part[0].src;
                const int32_t *rows = p.part[0].rows, *columns = p.part[0].columns;
                uint32_t begin = 0, units = p.part[0].units, H = p.part[0].H, W = p.part[0].W;
#pragma unroll
                for (int k = 1; k < kMaxResizedConcatInputs; ++k) {
                    if (p.part[k].units != 0 && u >= p.part[k].begin) {
                        src = p.part[k].src, rows = p.part[k].rows, columns = p.part[k].columns;
                        begin = p.part[k].begin, units = p.part[k].units, H = p.part[k].H, W = p.part[k].W;
                    }
                }
                int64_t from = pixel;
                if (rows != nullptr) {
                    const uint32_t line = fastDiv(pixel, p.divOW), ox = pixel - line * p.divOW.d;
                    const uint32_t n = fastDiv(line, p.divOH), oy = line - n * p.divOH.d;
                    const int32_t y = __ldg(rows + oy), x = __ldg(columns + ox);
                    from = (y | x) < 0 ? -1 : (int64_t(n) * H + y) * W + x;
                }
                if (from >= 0) {
                    v[j] = reinterpret_cast<const UNIT *>(src)[from * units + (u - begin)];
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint64_t at = first + uint64_t(j) * step;
            if (at < p.units) {
                reinterpret_cast<UNIT *>(out)[at] = v[j];
            }
        }
    }
}

// ---- ARGMAX along the last axis (argmax.comp:26-66): first strictly greater value wins, start = lowest, index 0 -----
// Rows of at most kArgmaxStage bytes: a block stages the contiguous bytes of its 256 rows in shared memory with wide
// loads, then a thread scans a row there.  Longer rows: a warp per row, the smallest index among equal maxima.
// 129 600 rows of 21 bytes (a per-pixel classifier): 20.5 -> 7.1 us.
constexpr int kArgmaxStage = 128;

template <typename T>
__global__ void __launch_bounds__(256)
    argmaxShortKernel(const T *in, int32_t *out, int64_t rows, int len, int32_t lowest) {
    dependencySync();
    __shared__ __align__(16) uint8_t stage[256 * kArgmaxStage];
    const int64_t total = rows * len * int64_t(sizeof(T));
    for (int64_t row0 = int64_t(blockIdx.x) * 256; row0 < rows; row0 += int64_t(gridDim.x) * 256) {
        const int64_t base = row0 * len * int64_t(sizeof(T)); // a multiple of 256 bytes
        const int bytes = int(min(int64_t(256) * len * int64_t(sizeof(T)), total - base));
        const uint8_t *src = reinterpret_cast<const uint8_t *>(in) + base;
        __syncthreads();
        for (int i = threadIdx.x * 16; i + 16 <= bytes; i += 256 * 16) {
            *reinterpret_cast<uint4 *>(stage + i) = *reinterpret_cast<const uint4 *>(src + i);
        }
        if (int(threadIdx.x) < (bytes & 15)) {
            stage[(bytes & ~15) + threadIdx.x] = src[(bytes & ~15) + threadIdx.x];
        }
        __syncthreads();
        if (row0 + threadIdx.x < rows) {
            const T *row = reinterpret_cast<const T *>(stage) + threadIdx.x * len;
            int32_t best = lowest, bestIndex = 0;
            for (int k = 0; k < len; ++k) {
                const int32_t v = int32_t(row[k]);
                if (v > best) {
                    best = v;
                    bestIndex = k;
                }
            }
            out[row0 + threadIdx.x] = bestIndex;
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(256)
    argmaxLongKernel(const T *in, int32_t *out, int64_t rows, int len, int32_t lowest) {
    dependencySync();
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t(gridDim.x) * blockDim.x) >> 5;
    for (int64_t row = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; row < rows; row += warps) {
        const T *src = in + row * len;
        int32_t best = lowest, bestIndex = 0x7fffffff; // a lane that saw nothing above the start loses every tie
        for (int k = lane; k < len; k += 32) {
            const int32_t v = int32_t(src[k]);
            if (v > best) {
                best = v;
                bestIndex = k;
            }
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            const int32_t v = __shfl_xor_sync(0xffffffffu, best, d), i = __shfl_xor_sync(0xffffffffu, bestIndex, d);
            if (v > best || (v == best && i < bestIndex)) {
                best = v;
                bestIndex = i;
            }
        }
        if (lane == 0) {
            out[row] = bestIndex == 0x7fffffff ? 0 : bestIndex;
        }
    }
}

template <typename T>
int launchArgmax(const TView &in, const TView &out, int64_t rows, int len, cudaStream_t s) {
    const T *pi = reinterpret_cast<const T *>(in.ptr);
    int32_t *po = reinterpret_cast<int32_t *>(out.ptr);
    const int32_t lowest = int32_t(typeLowest(in.dtype));
    if (len * int(sizeof(T)) <= kArgmaxStage) {
        launchOverlapped(argmaxShortKernel<T>, dim3(gridFor(rows, 256, 16)), 256, 0, s, pi, po, rows, len, lowest);
    } else {
        launchOverlapped(argmaxLongKernel<T>, dim3(gridFor(rows * 32, 256, 16)), 256, 0, s, pi, po, rows, len, lowest);
    }
    return finish("ARGMAX");
}

bool packedTensor(const TView &t) {
    int64_t st = dtypeSize(t.dtype);
    for (int i = t.rank - 1; i >= 0; --i) {
        if (t.strides[i] != st) {
            return false;
        }
        st *= t.dims[i];
    }
    return st > 0;
}

} // namespace

// Rule: two axes of at least eight elements that trade the last place go through tiles, everything else as runs (a
// transpose that keeps the last axis has long ones, and a very thin matrix would leave most of a tile idle).
bool moveTranspose(const TView &in, const TView &out, const uint32_t *perms, cudaStream_t s, int *rc) {
    const int rank = out.rank;
    if (!sameElement(in, out) || rank < 1) {
        return false;
    }
    const int64_t elem = dtypeSize(out.dtype), n = numelOf(out);
    uint32_t seen = 0;
    for (int i = 0; i < rank; ++i) {
        if (perms[i] >= uint32_t(rank) || in.dims[perms[i]] != out.dims[i]) {
            return false;
        }
        seen |= 1u << perms[i];
    }
    if (seen != (1u << rank) - 1u || n >= (int64_t(1) << 31) || n <= 0) {
        return false;
    }
    // where the input's last axis goes in the output
    int to = 0;
    while (int(perms[to]) != rank - 1) {
        ++to;
    }
    const uint32_t from = perms[rank - 1];
    if (to != rank - 1 && elem <= 4 && in.dims[from] >= 8 && in.dims[rank - 1] >= 8 && in.strides[rank - 1] == elem &&
        out.strides[rank - 1] == elem) {
        TileTranspose p{};
        p.R = int32_t(in.dims[from]), p.C = int32_t(in.dims[rank - 1]);
        p.srcRow = in.strides[from], p.dstRow = out.strides[to];
        int64_t matrices = 1;
        for (int i = 0; i < rank - 1; ++i) {
            if (i == to) {
                continue;
            }
            p.dims[p.axes] = makeFastDiv(out.dims[i]);
            p.srcStride[p.axes] = in.strides[perms[i]];
            p.dstStride[p.axes] = out.strides[i];
            ++p.axes;
            matrices *= out.dims[i];
        }
        const int64_t tilesC = (p.C + 63) / 64, perMatrix = tilesC * ((p.R + 63) / 64), tiles = matrices * perMatrix;
        const uintptr_t bits = reinterpret_cast<uintptr_t>(in.ptr) | reinterpret_cast<uintptr_t>(out.ptr);
        bool aligned = (bits & uintptr_t(elem - 1)) == 0;
        for (int i = 0; i < rank; ++i) {
            aligned = aligned && in.strides[i] % elem == 0 && out.strides[i] % elem == 0;
        }
        if (aligned && tiles < (int64_t(1) << 31)) {
            p.tilesC = makeFastDiv(tilesC);
            p.tilesPerMatrix = makeFastDiv(perMatrix);
            const int grid = int(std::min<int64_t>(tiles, int64_t(kNumSMs) * 8));
            const auto *pi = reinterpret_cast<const uint8_t *>(in.ptr);
            auto *po = reinterpret_cast<uint8_t *>(out.ptr);
            if (elem == 1) {
                launchOverlapped(tileTransposeKernel<uint8_t>, dim3(grid), 256, 0, s, pi, po, uint32_t(tiles), p);
            } else if (elem == 2) {
                launchOverlapped(tileTransposeKernel<uint16_t>, dim3(grid), 256, 0, s, pi, po, uint32_t(tiles), p);
            } else {
                launchOverlapped(tileTransposeKernel<uint32_t>, dim3(grid), 256, 0, s, pi, po, uint32_t(tiles), p);
            }
            *rc = finish("TRANSPOSE");
            return true;
        }
    }
    MoveAxes a;
    for (int i = 0; i < rank; ++i) {
        a.add(out.dims[i], in.strides[perms[i]], out.strides[i]);
    }
    return moveOne(a, elem, in.ptr, out.ptr, n, "TRANSPOSE", s, rc);
}

bool moveConcat(const TView *const *ins, const uint32_t *offsets, int count, const TView &out, uint32_t axis, cudaStream_t s,
                int *rc) {
    if (axis >= uint32_t(out.rank)) {
        return false;
    }
    const int64_t elem = dtypeSize(out.dtype);
    for (int first = 0; first < count; first += kMaxMoveParts) {
        const int n = std::min(kMaxMoveParts, count - first);
        RunMove parts[kMaxMoveParts];
        int64_t runs[kMaxMoveParts], bytes[kMaxMoveParts], unit = 16;
        for (int k = 0; k < n; ++k) {
            const TView &in = *ins[first + k];
            if (!sameElement(in, out) || numelOf(in) <= 0) {
                return false;
            }
            MoveAxes a;
            for (int i = 0; i < in.rank; ++i) {
                const int64_t end = int64_t(in.dims[i]) + (uint32_t(i) == axis ? offsets[first + k] : 0u);
                if (end > int64_t(out.dims[i])) {
                    return false; // the generic kernel drops what does not fit
                }
                a.add(in.dims[i], in.strides[i], out.strides[i]);
            }
            parts[k] = RunMove{};
            bytes[k] = numelOf(in) * elem;
            if (!makeRunMove(a, elem, in.ptr, out.ptr + int64_t(offsets[first + k]) * out.strides[axis], &parts[k], &runs[k],
                             &unit)) {
                return false;
            }
        }
        if (!launchRunMoves(parts, runs, bytes, n, unit, "CONCAT", s, rc)) {
            return false;
        }
        if (*rc != MLEL_SUCCESS) {
            return true;
        }
    }
    return true;
}

bool moveSlice(const TView &in, const TView &out, const uint32_t *start, cudaStream_t s, int *rc) {
    if (!sameElement(in, out)) {
        return false;
    }
    MoveAxes a;
    int64_t base = 0;
    for (int i = 0; i < out.rank; ++i) {
        if (int64_t(start[i]) + out.dims[i] > int64_t(in.dims[i])) {
            return false; // reads past the end are zeros: generic kernel
        }
        base += int64_t(start[i]) * in.strides[i];
        a.add(out.dims[i], in.strides[i], out.strides[i]);
    }
    return moveOne(a, dtypeSize(out.dtype), in.ptr + base, out.ptr, numelOf(out), "SLICE", s, rc);
}

bool moveTile(const TView &in, const TView &out, cudaStream_t s, int *rc) {
    if (!sameElement(in, out)) {
        return false;
    }
    MoveAxes a;
    for (int i = 0; i < out.rank; ++i) {
        if (in.dims[i] == 0 || out.dims[i] % in.dims[i] != 0) {
            return false;
        }
        a.add(out.dims[i] / in.dims[i], 0, int64_t(in.dims[i]) * out.strides[i]);
        a.add(in.dims[i], in.strides[i], out.strides[i]);
    }
    return moveOne(a, dtypeSize(out.dtype), in.ptr, out.ptr, numelOf(out), "TILE", s, rc);
}

bool moveReverse(const TView &in, const TView &out, uint32_t axis, cudaStream_t s, int *rc) {
    if (!sameElement(in, out) || axis >= uint32_t(out.rank)) {
        return false;
    }
    // the output walked forwards, the input backwards along `axis`
    MoveAxes a;
    for (int i = 0; i < out.rank; ++i) {
        if (in.dims[i] != out.dims[i] || out.dims[i] == 0) {
            return false;
        }
        a.add(out.dims[i], uint32_t(i) == axis ? -in.strides[i] : in.strides[i], out.strides[i]);
    }
    return moveOne(a, dtypeSize(out.dtype), in.ptr + int64_t(in.dims[axis] - 1) * in.strides[axis], out.ptr, numelOf(out),
                   "REVERSE", s, rc);
}

int concatResized(const ResizedConcat &plan, const TView *const *ins, int count, const TView *tensors, const TView &out, cudaStream_t s) {
    const int64_t elem = dtypeSize(out.dtype), pixels = int64_t(out.dims[0]) * out.dims[1] * out.dims[2], pixelBytes = int64_t(out.dims[3]) * elem;
    uint64_t bits = uint64_t(pixelBytes) | reinterpret_cast<uintptr_t>(out.ptr);
    for (int k = 0; k < count; ++k) {
        bits |= uint64_t(ins[k]->dims[3]) * uint64_t(elem) | reinterpret_cast<uintptr_t>(ins[k]->ptr);
    }
    int64_t unit = 16;
    while ((bits & uint64_t(unit - 1)) != 0) {
        unit >>= 1;
    }
    ConcatParts p{};
    for (int k = 0; k < count; ++k) {
        ConcatPart &part = p.part[k];
        part.src = reinterpret_cast<const uint8_t *>(ins[k]->ptr);
        part.begin = uint32_t(plan.firstChannel[size_t(k)] * elem / unit), part.units = uint32_t(ins[k]->dims[3] * elem / unit);
        part.H = ins[k]->dims[1], part.W = ins[k]->dims[2];
        if (plan.sources[size_t(k)] >= 0) {
            part.rows = reinterpret_cast<const int32_t *>(tensors[plan.sources[size_t(k)]].ptr);
            part.columns = part.rows + out.dims[1];
        }
    }
    p.units = uint32_t(pixels * pixelBytes / unit); // (below 2^31: GraphPipeline::fuseResizedConcats)
    p.perPixel = makeFastDiv(pixelBytes / unit), p.divOW = makeFastDiv(out.dims[2]), p.divOH = makeFastDiv(out.dims[1]);
    const dim3 grid(unsigned(gridFor((int64_t(p.units) + 3) / 4, kThreads, 16)));
    uint8_t *to = reinterpret_cast<uint8_t *>(out.ptr);
    const auto launch = [&](auto tag) { launchOverlapped(concatResizedKernel<decltype(tag)>, grid, kThreads, 0, s, to, p); };
    switch (unit) {
    case 16:
        launch(uint4{});
        break;
    case 8:
        launch(uint2{});
        break;
    case 4:
        launch(uint32_t{});
        break;
    case 2:
        launch(uint16_t{});
        break;
    default:
        launch(uint8_t{});
        break;
    }
    return finish("RESIZE+CONCAT");
}

bool moveResizeNearest(const TView &in, const TView &out, const ResizeAttr &a, cudaStream_t s, int *rc) {
    if (a.mode != 1 || in.rank != 4 || out.rank != 4 || in.dtype != out.dtype || !packedTensor(in) || !packedTensor(out) ||
        in.dims[0] != out.dims[0] || in.dims[3] != out.dims[3] || a.scale[0] <= 0 || a.scale[2] <= 0) {
        return false;
    }
    const int64_t pixelBytes = int64_t(in.dims[3]) * dtypeSize(in.dtype), bytes = numelOf(out) * dtypeSize(out.dtype);
    int64_t unit = 16;
    const uint64_t bits =
        uint64_t(pixelBytes) | reinterpret_cast<uintptr_t>(in.ptr) | reinterpret_cast<uintptr_t>(out.ptr);
    while ((bits & uint64_t(unit - 1)) != 0) {
        unit >>= 1;
    }
    const int64_t units = bytes / unit;
    if (units <= 0 || units >= (int64_t(1) << 31)) {
        return false;
    }
    const int grid = gridFor(units, kThreads, 16);
    const FastDiv perPixel = makeFastDiv(pixelBytes / unit), divOW = makeFastDiv(out.dims[2]), divOH = makeFastDiv(out.dims[1]);
    const auto launch = [&](auto tag) {
        launchOverlapped(resizeNearestKernel<decltype(tag)>, dim3(grid), kThreads, 0, s, reinterpret_cast<const uint8_t *>(in.ptr),
                         reinterpret_cast<uint8_t *>(out.ptr), uint32_t(units), perPixel, divOW, divOH, in.dims[1], in.dims[2], a);
    };
    switch (unit) {
    case 16:
        launch(uint4{});
        break;
    case 8:
        launch(uint2{});
        break;
    case 4:
        launch(uint32_t{});
        break;
    case 2:
        launch(uint16_t{});
        break;
    default:
        launch(uint8_t{});
        break;
    }
    *rc = finish("RESIZE");
    return true;
}

bool moveArgmaxLast(const TView &in, const TView &out, uint32_t axis, cudaStream_t s, int *rc) {
    if (in.rank < 1 || int(axis) != in.rank - 1 || out.rank != in.rank - 1 || out.dtype != MLEL_I32 || !packedTensor(in) ||
        !packedTensor(out) || (reinterpret_cast<uintptr_t>(in.ptr) & 15u) != 0) {
        return false;
    }
    const int64_t len = in.dims[axis], rows = numelOf(out);
    if (len <= 0 || len >= (int64_t(1) << 30) || rows <= 0 || rows * len != numelOf(in)) {
        return false;
    }
    if (in.dtype == MLEL_I8) {
        *rc = launchArgmax<int8_t>(in, out, rows, int(len), s);
    } else if (in.dtype == MLEL_I16) {
        *rc = launchArgmax<int16_t>(in, out, rows, int(len), s);
    } else if (in.dtype == MLEL_I32) {
        *rc = launchArgmax<int32_t>(in, out, rows, int(len), s);
    } else {
        return false;
    }
    return true;
}

} // namespace mlel
