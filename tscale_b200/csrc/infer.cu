// One-token inference step of the int8 model over a batch of sequences with per-layer int8 KV caches.  Replaces NCPUInfer::ComputePrediction / AddLookupProduct of the reference
// (code/gpt/train/cpu_infer.cpp:466-560), which runs one sequence on the CPU, by a batch of sequences on the GPU:
//
//   state = sum of label embeddings * scale                                    (cpu_infer.cpp:536-543)
//   per layer (cpu_infer.cpp:466-527):
//     norm   = NormalizeState(state, tiles of 128)            -> int8
//     qk, qv, k, v = int8 matrix * norm (exact int32), rope on qk and qv, NormalizeState per head -> int8
//     cache.append(qv, qvScale * QVScale * VEC_SCALE * dotScale(dim), v);  val = decode attention(qk, cache)
//     kv     = int8(k[z ^ blk] * val[z]), 4 blocks per head; state += Combiner * kv * scale
//     norm   = NormalizeState(state);  relu = max(0, NormalizeState(Expand * norm, per head));  state += Contract * relu * scale
//   prediction = softmax2(FinalLayer * NormalizeState(state) * scale + bias)    (cpu_infer.cpp:549-558)
//
// The layers are one persistent kernel (infer_persistent.cu); here are the final layer, the softmax and the entry points.  Everything but
// the attention weights and the last softmax is integer or single-rounded float arithmetic in the reference's order (sums of squares
// are accumulated sequentially like the scalar loops there), so those stages are bit-identical to the CPU code; the attention and the
// softmax use exp2 instead of the CPU's polynomial.  The matrix products read every int8 weight once per step for the whole batch (tcgen05
// kind::i8, exact int32 accumulators).
#include "att_sm100_common.cuh"
#include "infer_internal.cuh"

namespace tsa {

// ---- the final layer ------------------------------------------------------------------------------------------------
// logits[b][r] = (float)(int32 dot of vec[b] and W[r])   (MulForward, cpu_infer.cpp:282-293)
// One CTA = 128 rows of the matrix times all sequences (at most 64): tcgen05.mma kind::i8, M = 128 matrix rows, N = 64 sequences,
// exact int32 accumulators in 64 tensor-memory columns.  Thread 0 streams the row slab and the batch's vectors through a ring of
// GEMM_STAGES shared-memory stages of 128 columns (TMA, 128-byte swizzle; rows past the matrix and sequences past the batch read as
// zeros) and issues the MMAs; afterwards thread t holds row t of the tile and writes its products, coalesced over the rows of a
// warp.  Two CTAs per SM, so that one's epilogue runs under the other's stream.  The rows do not depend on the layers before: the
// first GEMM_STAGES slabs are requested before the wait for them (dependent launch).  Every wait is bounded.
constexpr int GEMM_STAGES = 4;
constexpr int GEMM_M = 128, GEMM_N = 64, GEMM_KB = 128;
constexpr int GEMM_STAGE_BYTES = (GEMM_M + GEMM_N) * GEMM_KB;
constexpr int GEMM_SMEM_BYTES = GEMM_STAGES * GEMM_STAGE_BYTES + 1024 /* barriers */ + 1024 /* alignment */;

struct TGemmMisc {
    uint64_t Full[GEMM_STAGES], Empty[GEMM_STAGES], Done;
    uint32_t TmemBase;
};

__global__ void __launch_bounds__(128, 2) InferGemmI8Kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmVec, float *out,
    int rows, int nSeq, int chunks, int *status)
{
    constexpr uint32_t IDESC = MakeInstrDesc(2, 1, 1, 0, 0, GEMM_M, GEMM_N); // s32 accumulators, s8 x s8, both K-major
    extern __shared__ uint8_t gemmSmemRaw[];
    const int rowBase = blockIdx.x * GEMM_M;
    uint8_t *smem = (uint8_t *)(((uintptr_t)gemmSmemRaw + 1023) & ~(uintptr_t)1023);
    TGemmMisc &misc = *reinterpret_cast<TGemmMisc *>(smem + GEMM_STAGES * GEMM_STAGE_BYTES);
    const int tid = threadIdx.x, warp = tid >> 5;
    if (tid == 0) {
#pragma unroll
        for (int s = 0; s < GEMM_STAGES; ++s) {
            MbarInit(&misc.Full[s], 1);
            MbarInit(&misc.Empty[s], 1);
        }
        MbarInit(&misc.Done, 1);
        FenceBarrierInit();
    }
    if (warp == 0) {
        TmemAlloc(&misc.TmemBase, GEMM_N);
        TmemRelinquish();
    }
    TcFenceBefore();
    __syncthreads();
    TcFenceAfter();
    PdlTrigger();
    const uint32_t tmem = misc.TmemBase;
    bool failed = false;
    if (tid == 0) {
        PrefetchTensorMap(&tmW);
        PrefetchTensorMap(&tmVec);
        auto slab = [&](int chunk) {
            const int s = chunk % GEMM_STAGES;
            MbarExpectTx(&misc.Full[s], GEMM_STAGE_BYTES);
            TmaLoad2D(smem + s * GEMM_STAGE_BYTES, &tmW, chunk * GEMM_KB, rowBase, &misc.Full[s]);
        };
        auto vectors = [&](int chunk) {
            const int s = chunk % GEMM_STAGES;
            TmaLoad2D(smem + s * GEMM_STAGE_BYTES + GEMM_M * GEMM_KB, &tmVec, chunk * GEMM_KB, 0, &misc.Full[s]);
        };
        int issued = 0, landed = 0; // chunks requested / chunks whose copies were seen to arrive
        for (int c = 0; c < GEMM_STAGES && c < chunks; ++c) {
            slab(c);
        }
        PdlWait();
        for (int c = 0; c < GEMM_STAGES && c < chunks; ++c) {
            vectors(c);
            ++issued;
        }
        for (int c = 0; c < chunks && !failed; ++c) {
            const int s = c % GEMM_STAGES;
            if (!WaitBar(&misc.Full[s], (uint32_t)((c / GEMM_STAGES) & 1))) {
                failed = true;
                if (status) {
                    atomicOr(status, kDevTimeoutTma);
                }
                break;
            }
            ++landed;
            TcFenceAfter();
            const uint32_t sA = SmemAddr(smem + s * GEMM_STAGE_BYTES), sB = sA + GEMM_M * GEMM_KB;
#pragma unroll
            for (int ks = 0; ks < GEMM_KB / 32; ++ks) {
                const uint64_t aDesc = MakeSmemDesc(sA + ks * 32, 16, 8 * GEMM_KB, 128);
                const uint64_t bDesc = MakeSmemDesc(sB + ks * 32, 16, 8 * GEMM_KB, 128);
                MmaI8SS(tmem, aDesc, bDesc, IDESC, (c > 0 || ks > 0) ? 1u : 0u);
            }
            MmaCommit(&misc.Empty[s]);
            // the stage of the chunk before this one has long been read (waiting for this chunk's own products would stall the
            // stream on every commit round trip)
            const int ahead = c - 1 + GEMM_STAGES;
            if (c > 0 && ahead < chunks) {
                if (!WaitBar(&misc.Empty[ahead % GEMM_STAGES], (uint32_t)(((c - 1) / GEMM_STAGES) & 1))) {
                    failed = true; // the MMAs that read this stage never finished
                    if (status) {
                        atomicOr(status, kDevTimeoutMma);
                    }
                    break;
                }
                slab(ahead);
                vectors(ahead);
                ++issued;
            }
        }
        if (failed) {
            // copies that were requested but never consumed must not land after the CTA is gone: wait (bounded) for them
            for (int t = landed; t < issued; ++t) {
                WaitBar(&misc.Full[t % GEMM_STAGES], (uint32_t)((t / GEMM_STAGES) & 1));
            }
        }
        MmaCommit(&misc.Done);
    } else {
        PdlWait();
    }
    if (!WaitBar(&misc.Done, 0)) {
        failed = true;
        if (status) {
            atomicOr(status, kDevTimeoutMma);
        }
    }
    TcFenceAfter();
    failed = __syncthreads_or(failed ? 1 : 0) != 0;
    const int row = rowBase + tid;
    const uint32_t tLane = tmem + ((uint32_t)(warp * 32) << 16);
#pragma unroll 1
    for (int c0 = 0; c0 < GEMM_N && c0 < nSeq; c0 += 32) {
        uint32_t accum[32];
        TmemLd32(tLane + c0, accum);
        TmemWaitLd();
        if (!failed && row < rows) {
#pragma unroll
            for (int cc = 0; cc < 32; ++cc) {
                if (c0 + cc < nSeq) {
                    out[(size_t)(c0 + cc) * rows + row] = (float)(int)accum[cc];
                }
            }
        }
    }
    TcFenceBefore();
    __syncthreads();
    if (warp == 0) {
        TmemDealloc(tmem, GEMM_N);
    }
}

// SoftMax of the final layer (cpu_infer.cpp:340-354): base 2, the maximum starts at 0 (TSoftMaxBuf::Clear).
// Two kernels over (sequence, slice of the vocabulary) so that a batch of 64 sequences fills the GPU: the first leaves
// each slice's maximum and sum of 2^(w - max), the second merges the slices' pairs and writes the probabilities.
constexpr int INF_SOFTMAX_SLICES = 64;

__device__ __forceinline__ float BlockReduce(float v, bool isMax, float *red)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    v = isMax ? WarpMax(v) : WarpSum(v);
    __syncthreads(); // red may still be read from the previous reduction
    if (lane == 0) {
        red[warp] = v;
    }
    __syncthreads();
    float r = red[0];
    for (int w = 1; w < warps; ++w) {
        r = isMax ? fmaxf(r, red[w]) : r + red[w];
    }
    return r;
}

__global__ void __launch_bounds__(256) InferSoftmaxPartKernel(const float *logits, const float *bias, float finalScale, int vocab, float *part)
{
    __shared__ float red[8];
    PdlTrigger();
    PdlWait();
    const int b = blockIdx.y, slice = blockIdx.x;
    const int per = (vocab + INF_SOFTMAX_SLICES - 1) / INF_SOFTMAX_SLICES;
    const int x0 = slice * per, x1 = min(x0 + per, vocab);
    const float *l = logits + (size_t)b * vocab;
    float mx = 0;
    for (int x = x0 + threadIdx.x; x < x1; x += blockDim.x) {
        mx = fmaxf(mx, __fadd_rn(__fmul_rn(l[x], finalScale), bias[x]));
    }
    mx = BlockReduce(mx, true, red);
    float sum = 0;
    for (int x = x0 + threadIdx.x; x < x1; x += blockDim.x) {
        sum += exp2f(__fadd_rn(__fmul_rn(l[x], finalScale), bias[x]) - mx);
    }
    sum = BlockReduce(sum, false, red);
    if (threadIdx.x == 0) {
        part[(b * INF_SOFTMAX_SLICES + slice) * 2] = mx;
        part[(b * INF_SOFTMAX_SLICES + slice) * 2 + 1] = sum;
    }
}

__global__ void __launch_bounds__(256) InferSoftmaxKernel(const float *logits, const float *bias, float finalScale, int vocab, const float *part,
    float *prediction)
{
    PdlTrigger();
    PdlWait();
    const int b = blockIdx.y, slice = blockIdx.x;
    const int per = (vocab + INF_SOFTMAX_SLICES - 1) / INF_SOFTMAX_SLICES;
    const int x0 = slice * per, x1 = min(x0 + per, vocab);
    // the slices' pairs, one per thread
    __shared__ float red[8];
    const bool has = threadIdx.x < INF_SOFTMAX_SLICES;
    const float2 pair = has ? *reinterpret_cast<const float2 *>(part + (b * INF_SOFTMAX_SLICES + threadIdx.x) * 2) : make_float2(0.0f, 0.0f);
    const float mx = BlockReduce(pair.x, true, red);
    const float sum = BlockReduce(has ? pair.y * exp2f(pair.x - mx) : 0.0f, false, red);
    const float inv = 1.0f / sum;
    const float *l = logits + (size_t)b * vocab;
    float *out = prediction + (size_t)b * vocab;
    for (int x = x0 + threadIdx.x; x < x1; x += blockDim.x) {
        out[x] = exp2f(__fadd_rn(__fmul_rn(l[x], finalScale), bias[x]) - mx) * inv;
    }
}

static int LaunchFinalLayer(const signed char *matrix, int rows, int cols, const int8_t *vec, int nSeq, float *logits, int *statusWord, cudaStream_t stream)
{
    CUtensorMap mw, mv;
    tsa_ptr2d w = {(void *)matrix, cols, cols, rows}, v = {(void *)vec, cols, cols, nSeq};
    int rc = MakeTileMapEx(&mw, w, 1, GEMM_KB, GEMM_M, "final layer");
    if (rc == TSA_OK) {
        rc = MakeTileMapEx(&mv, v, 1, GEMM_KB, GEMM_N, "inference vectors");
    }
    const void *kern = (const void *)InferGemmI8Kernel;
    if (rc == TSA_OK) {
        rc = CheckCuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GEMM_SMEM_BYTES), "cudaFuncSetAttribute");
    }
    if (rc != TSA_OK) {
        return rc;
    }
    int chunks = cols / GEMM_KB;
    void *args[] = {&mw, &mv, &logits, &rows, &nSeq, &chunks, &statusWord};
    return CheckCuda(LaunchPdl(kern, dim3((rows + GEMM_M - 1) / GEMM_M), dim3(128), GEMM_SMEM_BYTES, stream, args), "final layer launch");
}

static size_t Align256(size_t x)
{
    return (x + 255) / 256 * 256;
}

TInferBuffers CarveInferBuffers(const tsa_infer_model *m, int nSeq, void *base)
{
    const tsa_infer_dims &d = m->dims;
    const size_t hs = (size_t)d.head_count * d.head_dim;
    const int perGroup = AttGroupHeads(d.head_count, d.head_dim), headGroups = (d.head_count + perGroup - 1) / perGroup;
    TInferBuffers b;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        void *p = base ? (char *)base + off : nullptr;
        off += Align256(bytes);
        return p;
    };
    b.Sync = (int *)take(sizeof(int) * (64 + (size_t)nSeq * headGroups));
    b.Proj = (int *)take(sizeof(int) * nSeq * 4 * hs);
    b.Comb = (int *)take(sizeof(int) * nSeq * d.dim);
    b.Expand = (int *)take(sizeof(int) * nSeq * d.relu_dim);
    b.Contract = (int *)take(sizeof(int) * nSeq * d.dim);
    b.ZeroBytes = off;
    b.StateA = (float *)take(sizeof(float) * nSeq * d.dim);
    b.StateB = (float *)take(sizeof(float) * nSeq * d.dim);
    b.Logits = (float *)take(sizeof(float) * nSeq * d.vocab_size);
    b.SoftmaxPart = (float *)take(sizeof(float) * nSeq * INF_SOFTMAX_SLICES * 2);
    b.NormState = (int8_t *)take((size_t)nSeq * d.dim);
    b.K8 = (int8_t *)take((size_t)nSeq * hs);
    b.Kv8 = (int8_t *)take((size_t)nSeq * hs * 4);
    // partials of the attention's chunks
    b.Partial = (float *)take(sizeof(float) * ((size_t)INF_MAX_CHUNKS + nSeq) * d.head_count * (d.head_dim + 4));
    b.Total = off;
    return b;
}

static int CheckInferModel(const tsa_infer_model *m, int nSeq, const char *fn)
{
    TSA_REQUIRE(m != nullptr, "%s: null model", fn);
    const tsa_infer_dims &d = m->dims;
    TSA_REQUIRE(d.head_dim == 64 || d.head_dim == 128, "%s: head_dim %d must be 64 or 128 (query and value heads have one size here)", fn, d.head_dim);
    TSA_REQUIRE(d.dim > 0 && d.dim % INF_NORM_TILE == 0, "%s: dim %d must be a multiple of %d", fn, d.dim, INF_NORM_TILE);
    TSA_REQUIRE(d.head_count > 0 && d.relu_dim > 0 && d.relu_dim % d.head_count == 0 && d.relu_dim % GEMM_KB == 0,
        "%s: relu_dim %d must be a multiple of head_count %d and of %d", fn, d.relu_dim, d.head_count, GEMM_KB);
    TSA_REQUIRE(d.vocab_size > 0 && d.label_count > 0 && d.layer_count >= 0, "%s: vocab_size, label_count must be positive", fn);
    TSA_REQUIRE(nSeq >= 0 && nSeq <= INF_MAX_SEQ, "%s: %d sequences per step, at most %d", fn, nSeq, INF_MAX_SEQ);
    return TSA_OK;
}

} // namespace tsa

using namespace tsa;

extern "C" __attribute__((visibility("default"))) size_t tsa_infer_workspace_bytes(const tsa_infer_model *model, int nSeq, int maxCtx)
{
    if (CheckInferModel(model, nSeq, "tsa_infer_workspace_bytes") != TSA_OK || nSeq == 0 || maxCtx < 0) {
        return 0;
    }
    return CarveInferBuffers(model, nSeq, nullptr).Total;
}

extern "C" __attribute__((visibility("default"))) int tsa_infer_step(const tsa_infer_model *model, const tsa_kv_seq *const *layerSeqs, int *ctxLens,
    int capacity, const int *labels, int labelsPerSeq, int nSeq, int maxCtx, float *prediction, float *logits, void *workspace,
    size_t workspaceBytes, int *statusWord, tsa_stream_t streamArg)
{
    int rc = CheckInferModel(model, nSeq, "tsa_infer_step");
    if (rc != TSA_OK) {
        return rc;
    }
    if (nSeq == 0) {
        return TSA_OK;
    }
    const tsa_infer_dims &d = model->dims;
    TSA_REQUIRE(labels && ctxLens && labelsPerSeq > 0 && maxCtx >= 0 && capacity > maxCtx, "tsa_infer_step: labels, ctxLens, capacity > maxCtx");
    TSA_REQUIRE(d.layer_count == 0 || (model->layers && layerSeqs), "tsa_infer_step: null layers");
    TSA_REQUIRE(model->label_embed && model->final_layer && model->bias && model->rope && model->rope_len > maxCtx,
        "tsa_infer_step: model tables (the rope table must cover position maxCtx = %d, it has %d rows)", maxCtx, model->rope_len);
    for (int l = 0; l < d.layer_count; ++l) {
        const tsa_infer_layer &layer = model->layers[l];
        const void *matrices[7] = {layer.qk, layer.qv, layer.k, layer.v, layer.combiner, layer.expand, layer.contract};
        for (const void *m : matrices) {
            TSA_REQUIRE(m && layerSeqs[l], "tsa_infer_step: layer %d has a null matrix or cache", l);
            TSA_REQUIRE((uintptr_t)m % 16 == 0, "tsa_infer_step: a matrix of layer %d is not 16-byte aligned", l); // copied 16 bytes at a time
        }
        TSA_REQUIRE(layer.attention_width >= 0, "tsa_infer_step: layer %d has a negative attention width", l);
    }
    const TInferBuffers need = CarveInferBuffers(model, nSeq, nullptr);
    TSA_REQUIRE(workspace && workspaceBytes >= need.Total && (uintptr_t)workspace % 256 == 0, "tsa_infer_step: workspace of %zu bytes, 256-byte aligned, needed",
        need.Total);
    const TInferBuffers b = CarveInferBuffers(model, nSeq, workspace);
    cudaStream_t stream = (cudaStream_t)streamArg;
    const int dim = d.dim;
    rc = InferLayersPersistent(model, layerSeqs, ctxLens, capacity, labels, labelsPerSeq, nSeq, maxCtx, b, statusWord, stream);
    if (rc != TSA_OK) {
        return rc;
    }
    if (prediction || logits) {
        float *lg = logits ? logits : b.Logits;
        rc = LaunchFinalLayer(model->final_layer, d.vocab_size, dim, b.NormState, nSeq, lg, statusWord, stream);
        if (rc != TSA_OK) {
            return rc;
        }
        if (prediction) {
            // CalcDotScale(dim) * CalcFinalLayerMult() * FinalLayerScale * VEC_SCALE (cpu_infer.cpp:555)
            const float finalScale = sqrtf(1.0f / dim) * (1.0f / 0.693147f) * model->final_layer_scale * INF_VEC_SCALE;
            dim3 gridS(INF_SOFTMAX_SLICES, nSeq);
            const float *bias = model->bias;
            int vocab = d.vocab_size;
            void *args[] = {&lg, &bias, (void *)&finalScale, &vocab, (void *)&b.SoftmaxPart, &prediction};
            rc = CheckCuda(LaunchPdl((const void *)InferSoftmaxPartKernel, gridS, dim3(256), 0, stream, args), "inference softmax launch");
            if (rc == TSA_OK) {
                rc = CheckCuda(LaunchPdl((const void *)InferSoftmaxKernel, gridS, dim3(256), 0, stream, args), "inference softmax launch");
            }
        }
    }
    return rc;
}
