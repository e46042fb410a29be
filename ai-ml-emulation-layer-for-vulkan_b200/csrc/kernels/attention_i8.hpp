// Host description of a fused quantised attention (attention_i8.cu).
#pragma once

#include "device_common.cuh"

namespace mlel {

// Everything about the node that its graph fixes: shapes, strides and the RESCALE constants in the kernel's forms.
struct AttentionPlan {
    int32_t batches, heads; // batches = sequences x heads
    int32_t queries, keys, headDim;
    int64_t qStride[3], kStride[3], vStride[3], oStride[3]; // bytes: sequence, head, token (the head dimension is contiguous)
    int64_t qOffset, kOffset, vOffset; // bytes, of the first element in the operand's tensor (a multiple of 16)
    // first RESCALE (score differences, int32 -> int16), its result 32768 higher: max((x * mult + addend) >> 32 + shift, 0)
    int32_t diffMult, diffShift;
    int64_t diffAddend;
    // 4 and 0x8000, from the parameter block so that they stay operands of one multiply-add and one logic operation
    uint32_t entryBytes, unitByte;
    FastRescale denom; // row sums -> int16
    int32_t denomOutZp;
    int64_t mulRound; // MUL: (e * r + round) >> shift
    int32_t mulShift;
    // last RESCALE, minus the product's zero point, before saturation: (x * mult + addend) >> 32 + shift
    int32_t probMult, probShift;
    int64_t probAddend;
    bool narrow;       // both RESCALEs divided by a power of two of their multipliers: (x * mult + addend) >> shift in 32 bits
    bool unsignedProb;                      // zero point -128: probabilities are stored as unsigned bytes
    FastRescale context;
    int32_t contextOutZp;
};

// Limits of the kernel: a row of scores fits tensor memory (512 columns) and, with the operands, shared memory; below
// the second limit two blocks share an SM.
constexpr int kAttentionMaxKeys = 512, kAttentionTwoBlockKeys = 192;

int attentionFused(const AttentionPlan &plan, const TView &q, const TView &k, const TView &v, const TView &expTable,
                   const TView &recipTable, const TView &out, cudaStream_t s);
int attentionErrorWord();

} // namespace mlel
