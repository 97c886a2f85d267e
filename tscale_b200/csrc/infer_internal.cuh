// Shared by the files of the token step: constants and scalar helpers in the reference's rounding order.
#pragma once
#include "tsa_common.cuh"

namespace tsa {

constexpr float INF_VEC_SCALE = 1.0f / 24; // VEC_SCALE, cpu_infer.cpp:16
constexpr int INF_NORM_TILE = 128;         // STATE_NORM_TILE, model_dim.h:23
constexpr int INF_MAX_SEQ = 64;            // sequences per step
constexpr int INF_MAX_CHUNKS = 1024;       // chunks the keys of a layer are cut into, beside one per sequence

// ConvertToInt8 (cpu_infer.cpp:88-92): round to nearest even, clamp to +-127
__device__ __forceinline__ int ToInt8Clamp127(float x)
{
    return max(-127, min(127, __float2int_rn(x)));
}

// discrScale and 1 / discrScale of NormalizeState (cpu_infer.cpp:381-383); both 0 for an all-zero group
__device__ __forceinline__ void NormScales(float sum2, int n, float *discr, float *mult)
{
    if (sum2 == 0) {
        *discr = 0;
        *mult = 0;
    } else {
        const float sko = __fsqrt_rn(__fdiv_rn(sum2, (float)n));
        *discr = __fmul_rn(sko, INF_VEC_SCALE);
        *mult = __fdiv_rn(1.0f, *discr);
    }
}

// adds the squares of four consecutive elements in index order, one rounding per product and per sum
__device__ __forceinline__ float AddSquares(float sum2, float4 v)
{
    sum2 = __fadd_rn(sum2, __fmul_rn(v.x, v.x));
    sum2 = __fadd_rn(sum2, __fmul_rn(v.y, v.y));
    sum2 = __fadd_rn(sum2, __fmul_rn(v.z, v.z));
    return __fadd_rn(sum2, __fmul_rn(v.w, v.w));
}

// Heads the attention of the step takes together.  A warp-wide 16-byte load covers 512 columns: some heads of one stream of keys, or,
// with fewer heads, those of several streams.  Taken: the size that needs the fewest loads for a token's row (12 heads of 64: three groups
// of four heads, two streams per load, instead of eight and four heads or twice six with idle lanes), the largest of those.
inline int AttGroupHeads(int heads, int headDim)
{
    const int most = 512 / headDim;
    int best = 1;
    for (int g = 1; g <= most && g <= heads; ++g) {
        const int groups = (heads + g - 1) / g, bestGroups = (heads + best - 1) / best;
        if (groups * (most / best) <= bestGroups * (most / g)) { // groups / streams per load, cross-multiplied
            best = g;
        }
    }
    return best;
}

struct TInferBuffers {
    float *StateA, *StateB, *Logits, *SoftmaxPart, *Partial;
    int *Sync;      // grid barrier (64 words), counters of chunks done, then the int32 sums: zeroed before every step
    size_t ZeroBytes;
    int *Proj, *Comb, *Expand, *Contract;
    int8_t *NormState, *K8, *Kv8;
    size_t Total;
};

TInferBuffers CarveInferBuffers(const tsa_infer_model *m, int nSeq, void *base);

// all layers of the step: embedding to the normalised int8 state in b.NormState, caches appended and counted
int InferLayersPersistent(const tsa_infer_model *model, const tsa_kv_seq *const *layerSeqs, int *ctxLens, int capacity, const int *labels, int labelsPerSeq,
    int nSeq, int maxCtx, const TInferBuffers &b, int *statusWord, cudaStream_t stream);

} // namespace tsa
