// Depthwise 3x3 convolution with RESCALE from a table of per-channel constants (depthwise_i8.cu).
#pragma once

#include <cstdint>
#include <vector>

#include "kernels.hpp"

namespace mlel {

// What the kernel needs of one channel: two 16-byte words.
struct alignas(16) DepthwiseChannel {
    uint32_t weights[3]; // of a window row: bytes kx = 0, 1, 2
    int32_t start;       // of the sum: bias - input zero point * sum of weights - zero point of the RESCALE
    // result = ((sum * mult + addend) >> 32) >> shift.  The addend's words first: a pair of registers has to start at an even
    // one, in another place of a 16-byte load they are moved there for every result.
    uint32_t low, high; // rounding, output zero point
    int32_t mult, shift;
};
struct alignas(16) DepthwiseWord {
    uint32_t v[4];
};
static_assert(sizeof(DepthwiseChannel) == 2 * sizeof(DepthwiseWord), "read as two 16-byte words");

struct DepthwiseConstants {
    const int8_t *weights; // [3][3][channels]
    const int32_t *bias, *mult;
    const int8_t *shift;
    int32_t channels, biasCount, perChannel, doubleRound;
    int32_t inputZp, rescaleZp, outZp, lo;
};
// The table: for groups of four channels, word 2 k + h of group g is half h of channel 4 g + k and stands at [2 k + h][g], so that
// neighbouring threads, which have neighbouring groups, read neighbouring words.
// False: not a table's case (shifts outside 33 to 50, 32 where the sign does not count; negative multipliers; sums that
// could leave int32).
bool makeDepthwiseChannels(const DepthwiseConstants &d, std::vector<DepthwiseWord> *out);
bool depthwiseTableTakes(const TView &in, const TView &out, const ConvAttr &a);
int depthwiseFromTable(const TView &in, const TView &table, const TView &out, const ConvAttr &a, const DevRescale &r, cudaStream_t s);

} // namespace mlel
