// The layers of a token step as ONE persistent kernel: a cooperative launch with one CTA per SM whose phases are separated by
// grid-wide barriers.  What it computes is described in infer.cu; this file is about how.
//
// As separate launches the step was bound by launches and by latency, not by bytes: seven kernels per layer of 6 to 10 us each
// for matrices of 1 to 2 MB (680 us per token for one sequence, twelve layers; the weights stream in 20 us).  Here a layer is five
// phases
//     P  proj      += W_qk|qv|k|v * norm(state)         int32 sums, exact
//     A  attention     rope, per-head normalise, append to the caches, softmax(q K) V, times the combiner key -> int8
//     C  comb      += W_combiner * A
//     E  expand    += W_expand * norm(state + comb)
//     T  contract  += W_contract * relu(norm(expand))
// and a grid barrier (0.75 us: one counter, arrival and wait apart) behind each.  A matrix product is cut into items of one 128-row
// tile and some 128-column chunks, as many items as there are SMs, so that a 768 x 768 matrix uses the whole GPU; the items' int32 partial tiles are added in L2
// (red.add: exact, the order does not matter).  The consumer of a product forms its own input from those sums: every item of
// the next product normalises the 128-column chunk it multiplies with (a chunk is one STATE_NORM_TILE; the scalar loop's
// order of operations, so the codes are bit-identical to the CPU's), which costs each of them a few hundred nanoseconds and
// saves a phase and its barrier.  The weights do not depend on anything: every CTA keeps the tiles of its next items, across
// phases and layers, in flight in a ring of shared memory (cp.async), so that their DRAM latency is never on the path.
//
// Measured, twelve layers, dim 768, 12 heads x 64, vocabulary 50304, a whole token with the final layer and softmax, launches / graph:
//     1 sequence, 500 tokens of context       744 / 568 -> 323 us, of which 305 are there with windows of 64 tokens in all layers: sixty
//                                             phases at some 5 us, the barrier, the sums through L2 and the norm, in a chain; the
//                                             bytes take 20 us
//     64 sequences, 1024 to 8192 tokens       968 / 801 -> 707 / 701 us (three of four layers see 64 tokens): 439 us with the short
//                                             windows in all layers, and 89 us for every wide layer, whose keys and values then
//                                             stream at 5.5 TB/s
// Head counts whose chunks need a whole group of four warps leave a quarter of the groups a second unit: with 16 heads x 64 such a
// batch takes 975 / 968 us, where separate launches, 16 warps per SM in the attention, took 1085 / 897.
#include "att_sm100_common.cuh"
#include "decode_device.cuh"
#include "infer_internal.cuh"
#include <stddef.h>

namespace tsa {

// Attention works in groups of four warps.  Three of them leave the loop over keys the 168 registers it wants (64 of loads in flight); with
// a fourth, at 128, it spills and a token of 64 sequences takes 912 us where this takes 735.
constexpr int PS_THREADS = 384, PS_GROUPS = 3;
constexpr int PS_LOADERS = PS_THREADS - 32; // threads that request weight tiles: all but the warp whose first lane polls the grid barrier
constexpr int PS_RING = 8;                     // weight tiles in flight or in use per CTA
constexpr int PS_TILE = 128 * 128;             // bytes of a weight tile: 128 rows x 128 columns
constexpr int PS_B_BYTES = INF_MAX_SEQ * 128;  // the chunk's vectors, one row of 128 int8 per sequence
constexpr int PS_F_PITCH = 132;                // floats per row of the fp32 chunk: 16-byte rows that fall into different banks
constexpr int PS_MERGE_PITCH = 19;
constexpr int PS_STAGE_AHEAD = 3;              // quads of columns whose loads a thread has in flight (6: spills, +4 %)
constexpr int PS_LAYERS = 32;                  // layers per launch
constexpr int PS_CHUNKS_PER_SM = 4;            // the keys of a layer are cut into no more chunks than this times the SMs
constexpr int PS_MIN_CHUNK = 16;               // keys
constexpr long long PS_WAIT_CYCLES = 1ll << 31;

enum { PH_PROJ = 0, PH_COMB = 1, PH_EXPAND = 2, PH_CONTRACT = 3 };
enum { SRC_EMBED = 0, SRC_SUM = 1, SRC_STATE = 2 }; // where the first product of a launch gets the state from

struct TStepLayer {
    const int8_t *W[7]; // qk, qv, k, v, combiner, expand, contract
    const tsa_kv_seq *Seqs;
    int *CtxLens;
    float QvMult, CombScale, ContractScale, Slope;
    int Window;
};

struct TStepShape {
    int Tiles, Chunks; // 128-row tiles, 128-column chunks of the phase's matrices
    int Per, Splits;   // chunks per item, items per tile
};

struct TStepParams {
    TStepLayer Layers[PS_LAYERS];
    TStepShape Shape[4];
    int LayerCount, FirstSource;
    int NSeq, Dim, Heads, HeadSize, ReluDim, Capacity, MaxCtx, RopeLen;
    int HeadGroups, PerGroup;     // groups of heads the attention works in, heads of a group (the last may have fewer)
    int PerLoadLog;               // log2 of the streams of keys a warp-wide load covers
    int Split;                    // parts a chunk's keys are cut into, 1, 2 or 4
    const int *Labels;
    int LabelsPerSeq, LabelCount;
    const int8_t *Embed;
    float EmbedScale;
    const float *Rope;
    float DotScale;
    int *Barrier;                 // zero at launch
    int *Arrived;                 // [nSeq][head groups] chunks done of the rows that several units share, zero between uses
    int *Proj, *Comb, *Expand, *Contract; // int32 sums, zero at launch
    float *StateA, *StateB;
    int8_t *K8, *Kv8, *NormState;
    float *Partial;
    int *Status;
};

struct alignas(16) TAttGroupSmem {
    union {
        float Rot[4][8 * 68];     // projected vectors a warp works on (8 x 64 or 4 x 128), rotated; pitch D + 4 per head
        float Merge[4][32][PS_MERGE_PITCH]; // maximum, sum and 16 columns of every lane's stream of keys
    };
    float Mult[4][8];
    int8_t Q8[2048], K8[2048];    // codes of the queries and combiner keys, [sequence of the unit][heads of the group][D]
    int Last[2];                  // this unit is the last of the row's: its first sequence, its last one
};

// Units of the attention of one layer (see MakeAttPlan).
struct TAttPlan {
    int Window;                                // of the layer, -1: none yet
    int Chunk, Parts;                          // keys of a chunk, streams of keys it is worked on in
    int PerUnit, Slots;                        // chunks of a unit, and all of them
    int UnitBegin, UnitEnd;                    // this CTA's units
    int Pos[INF_MAX_SEQ];                      // position of each sequence's new token
    int Base[INF_MAX_SEQ], Count[INF_MAX_SEQ]; // its first chunk and their number
    uint8_t SeqOf[INF_MAX_CHUNKS + INF_MAX_SEQ]; // sequence of a chunk
};

// one 128 x 128 weight tile of the CTA's share of a layer
enum { TILE_FIRST = 1, TILE_LAST = 2 }; // of its item
struct TWeightTile {
    uint8_t Matrix, Flags; // index into TStepLayer::W
    uint16_t Chunk;
    int Tile;
};
constexpr int PS_TABLE = 512; // tiles per CTA and layer kept in shared memory (1.2 GB of weights in one layer); beyond it they are computed

// what the critical path reads of a layer
struct TLayerNow {
    float QvMult, CombScale, PrevContractScale, Slope;
    int Window;
};

struct TStepSmem {
    uint8_t Ring[PS_RING][PS_TILE];
    uint8_t B[PS_B_BYTES];
    union {
        struct {
            float F[INF_MAX_SEQ][PS_F_PITCH];
            float Mult[INF_MAX_SEQ];
        };
        TAttGroupSmem Att[PS_GROUPS];
    };
    TWeightTile Table[PS_TABLE];
    int PhaseBegin[5];            // first tile of each phase, and their number
    TAttPlan Plan[2];             // of the last two windows: the layers of a model alternate between two or so
    TLayerNow Now;                // of the present layer: a first read of a kernel parameter waits for the constant cache
    int PlanOf;                   // which of them is the present layer's
    tsa_kv_seq Seqs[INF_MAX_SEQ]; // the present layer's caches
    uint64_t MmaDone;
    uint32_t TmemBase;
    int Failed;
    int Passed;                   // arrivals at the grid barrier that complete its present phase
};

static_assert(sizeof(TAttGroupSmem) % 16 == 0 && offsetof(TAttGroupSmem, Q8) % 16 == 0 && offsetof(TAttGroupSmem, K8) % 16 == 0 && offsetof(TStepSmem, F) % 16 == 0 && offsetof(TStepSmem, B) % 1024 == 0,
    "16-byte accesses and swizzled operand tiles");
static_assert(sizeof(TStepSmem) + 1024 <= 227 * 1024, "shared memory of a CTA, with the slack that aligns the tiles");

__device__ __forceinline__ void CpAsync16(void *dst, const void *src, int bytes)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(SmemAddr(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void CpAsyncCommit()
{
    asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void CpAsyncWait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void GroupSync(int group)
{
    asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory");
}

// Barrier of the whole grid in two parts, so that what does not depend on the other CTAs runs between them.  One counter and one
// polling thread per CTA: 0.75 us when all arrive together (a flag per CTA polled by 148 threads took 3.1 us, eight counters 1.3).
// Bounded: the wait returns false in every thread of a CTA that has waited about a second.
__device__ __forceinline__ void GridArrive(const TStepParams &p)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(p.Barrier) : "memory");
    }
}
__device__ __forceinline__ bool GridWait(const TStepParams &p, TStepSmem &sm)
{
    if (threadIdx.x == 0) {
        const int passed = sm.Passed += gridDim.x;
        const long long t0 = clock64();
        int seen;
        for (;;) {
            asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(seen) : "l"(p.Barrier) : "memory");
            if (seen >= passed) {
                break;
            }
            if (clock64() - t0 > PS_WAIT_CYCLES) {
                sm.Failed = 1;
                if (p.Status) {
                    atomicOr(p.Status, kDevTimeoutMma);
                }
                break;
            }
        }
    }
    __syncthreads();
    return sm.Failed == 0;
}

// The CTA's weight tiles of one layer in the order it uses them, tile number `index`: item blockIdx.x, blockIdx.x + gridDim.x, ... of
// every phase, an item's chunks one after another.
__device__ __noinline__ TWeightTile ComputeTile(const TStepParams &p, int index)
{
    TWeightTile t = {};
    for (int phase = 0; phase < 4; ++phase) {
        const TStepShape &s = p.Shape[phase];
        for (int item = blockIdx.x; item < s.Tiles * s.Splits; item += gridDim.x) {
            const int tile = item / s.Splits, first = (item - tile * s.Splits) * s.Per, chunks = min(s.Per, s.Chunks - first);
            if (index < chunks) {
                const int perMatrix = phase == PH_PROJ ? s.Tiles / 4 : s.Tiles;
                t.Matrix = (uint8_t)(phase == PH_PROJ ? tile / perMatrix : phase + 3);
                t.Tile = tile % perMatrix;
                t.Chunk = first + index;
                t.Flags = (uint8_t)((index == 0 ? TILE_FIRST : 0) | (index == chunks - 1 ? TILE_LAST : 0));
                return t;
            }
            index -= chunks;
        }
    }
    return t;
}
__device__ __forceinline__ TWeightTile TileAt(const TStepParams &p, const TStepSmem &sm, int index)
{
    return index < PS_TABLE ? sm.Table[index] : ComputeTile(p, index);
}

// requests tile number `index` of layer l (nothing past the last layer) and closes the cp.async group; rows past the matrix read as
// zeros.  All warps but the first, whose lane polls the grid barrier meanwhile.
__device__ __forceinline__ void RequestTile(const TStepParams &p, const TStepSmem &sm, int l, int index, uint8_t *dst)
{
    if (l < p.LayerCount) {
        const TWeightTile t = TileAt(p, sm, index);
        const int8_t *w = p.Layers[l].W[t.Matrix];
        const TStepShape &s = p.Shape[t.Matrix < 4 ? PH_PROJ : t.Matrix - 3];
        const int rows = t.Matrix < 4 ? p.Heads * p.HeadSize : t.Matrix - 3 == PH_EXPAND ? p.ReluDim : p.Dim;
        const int pitch = s.Chunks * 128;
        w += (size_t)t.Tile * 128 * pitch + t.Chunk * 128;
#pragma unroll
        for (int k = 0; k < (PS_TILE / 16 + PS_LOADERS - 1) / PS_LOADERS; ++k) {
            const int idx = (int)threadIdx.x - 32 + k * PS_LOADERS, row = idx >> 3, c16 = idx & 7;
            if (idx < PS_TILE / 16) {
                const bool ok = t.Tile * 128 + row < rows;
                CpAsync16(dst + row * 128 + ((c16 ^ (row & 7)) << 4), ok ? w + (size_t)row * pitch + c16 * 16 : p.Layers[l].W[t.Matrix], ok ? 16 : 0);
            }
        }
    }
    CpAsyncCommit();
}

// Where the CTA stands in its sequence of weight tiles.
struct TTileCursor {
    int Used, Requested;      // tiles used up / requested so far, over all layers
    int NextLayer, NextIndex; // the next tile to request
};

// requests tiles until PS_RING - 1 of them are on their way or waiting (the slot of the tile used last is free again)
__device__ __noinline__ void RefillRing(const TStepParams &p, TStepSmem &sm, TTileCursor *cursor)
{
    TTileCursor c = *cursor;
#pragma unroll 1
    while (c.Requested - c.Used < PS_RING - 1) {
        if (threadIdx.x >= 32) {
            RequestTile(p, sm, c.NextLayer, c.NextIndex, sm.Ring[c.Requested % PS_RING]);
        }
        ++c.Requested;
        if (++c.NextIndex >= sm.PhaseBegin[4]) {
            c.NextIndex = 0;
            ++c.NextLayer;
        }
    }
    *cursor = c;
}

// one 16-byte piece (columns c16 * 16 ..) of row s of the operand tile, 128-byte swizzle
__device__ __forceinline__ void StoreCodes(uint8_t *tile, int s, int c16, int4 v)
{
    *reinterpret_cast<int4 *>(tile + s * 128 + ((c16 ^ (s & 7)) << 4)) = v;
}

// four columns of the sum of a token's label embeddings (cpu_infer.cpp:536-543)
__device__ __noinline__ float4 EmbedColumns(const TStepParams &p, int s, int col, bool report)
{
    float4 v = make_float4(0, 0, 0, 0);
    for (int k = 0; k < p.LabelsPerSeq; ++k) {
        const int label = p.Labels[s * p.LabelsPerSeq + k];
        if (label < 0 || label >= p.LabelCount) {
            if (col == 0 && report && p.Status) {
                atomicOr(p.Status, kDevBadSpan);
            }
            continue;
        }
        const int8_t *row = p.Embed + (size_t)label * p.Dim + col;
        const char4 e = ((uintptr_t)row & 3) == 0 ? *reinterpret_cast<const char4 *>(row) : make_char4(row[0], row[1], row[2], row[3]);
        v.x = __fadd_rn(v.x, __fmul_rn((float)e.x, p.EmbedScale));
        v.y = __fadd_rn(v.y, __fmul_rn((float)e.y, p.EmbedScale));
        v.z = __fadd_rn(v.z, __fmul_rn((float)e.z, p.EmbedScale));
        v.w = __fadd_rn(v.w, __fmul_rn((float)e.w, p.EmbedScale));
    }
    return v;
}

// columns [128 chunk, +128) of the state after the last update, in sm.F: source 0 = embedding, 1 = state + sums * scale, 2 = state.
// The writer also stores them to dst.  Ends with a barrier.
__device__ __forceinline__ void StageState(const TStepParams &p, TStepSmem &sm, int chunk, int source, const float *state, const int *sums, float scale, float *dst)
{
    if (source == SRC_EMBED) {
        for (int i = threadIdx.x; i < p.NSeq * 32; i += PS_THREADS) {
            const int s = i >> 5, x = (i & 31) * 4;
            const float4 e = EmbedColumns(p, s, chunk * 128 + x, dst != nullptr);
            *reinterpret_cast<float4 *>(&sm.F[s][x]) = e;
            if (dst) {
                *reinterpret_cast<float4 *>(dst + (size_t)s * p.Dim + chunk * 128 + x) = e;
            }
        }
        __syncthreads();
        return;
    }
    // a few quads of columns per thread and step, their loads before the first use (all of a thread's quads at once took the registers
    // the attention loop needs)
    constexpr int AHEAD = PS_STAGE_AHEAD;
#pragma unroll 1
    for (int base = threadIdx.x; base < p.NSeq * 32; base += AHEAD * PS_THREADS) {
        float4 v[AHEAD];
        int4 add[AHEAD];
#pragma unroll
        for (int k = 0; k < AHEAD; ++k) {
            const int i = base + k * PS_THREADS, s = i >> 5, col = chunk * 128 + (i & 31) * 4;
            if (i < p.NSeq * 32) {
                v[k] = __ldcg(reinterpret_cast<const float4 *>(state + (size_t)s * p.Dim + col));
                if (source == SRC_SUM) {
                    add[k] = __ldcg(reinterpret_cast<const int4 *>(sums + (size_t)s * p.Dim + col));
                }
            }
        }
#pragma unroll
        for (int k = 0; k < AHEAD; ++k) {
            const int i = base + k * PS_THREADS, s = i >> 5, x = (i & 31) * 4;
            if (i < p.NSeq * 32) {
                if (source == SRC_SUM) { // AddScaled, cpu_infer.cpp:296-303
                    v[k].x = __fadd_rn(v[k].x, __fmul_rn((float)add[k].x, scale));
                    v[k].y = __fadd_rn(v[k].y, __fmul_rn((float)add[k].y, scale));
                    v[k].z = __fadd_rn(v[k].z, __fmul_rn((float)add[k].z, scale));
                    v[k].w = __fadd_rn(v[k].w, __fmul_rn((float)add[k].w, scale));
                }
                *reinterpret_cast<float4 *>(&sm.F[s][x]) = v[k];
                if (dst) {
                    *reinterpret_cast<float4 *>(dst + (size_t)s * p.Dim + chunk * 128 + x) = v[k];
                }
            }
        }
    }
    __syncthreads();
}

// int8 codes of the staged columns [4 quad0, 4 (quad0 + quads)) under sm.Mult, into the operand tile; four columns per thread and step
// (sixteen left all but eight threads without work for one sequence and were four times the code)
__device__ __forceinline__ void QuantiseStaged(const TStepParams &p, TStepSmem &sm, int quad0, int quads, bool relu)
{
#pragma unroll 2
    for (int i = threadIdx.x; i < p.NSeq * 32; i += PS_THREADS) {
        const int s = i >> 5, x = (i & 31) * 4;
        if ((unsigned)((i & 31) - quad0) >= (unsigned)quads) {
            continue;
        }
        const float mult = sm.Mult[s];
        const float4 v = *reinterpret_cast<const float4 *>(&sm.F[s][x]);
        int q[4] = {ToInt8Clamp127(__fmul_rn(v.x, mult)), ToInt8Clamp127(__fmul_rn(v.y, mult)), ToInt8Clamp127(__fmul_rn(v.z, mult)),
            ToInt8Clamp127(__fmul_rn(v.w, mult))};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            q[j] = relu ? max(q[j], 0) : q[j];
        }
        const uint32_t w = (uint32_t)(q[0] & 0xff) | ((uint32_t)(q[1] & 0xff) << 8) | ((uint32_t)(q[2] & 0xff) << 16) | ((uint32_t)(q[3] & 0xff) << 24);
        *reinterpret_cast<uint32_t *>(sm.B + s * 128 + (((x >> 4) ^ (s & 7)) << 4) + (x & 15)) = w;
    }
}

// NormalizeState of the staged chunk (one STATE_NORM_TILE): one thread per sequence adds the squares in index order
__device__ __forceinline__ void NormaliseStaged(const TStepParams &p, TStepSmem &sm)
{
    const int s = threadIdx.x;
    if (s < p.NSeq) {
        float sum2 = 0;
#pragma unroll 8
        for (int x = 0; x < 128; x += 4) {
            sum2 = AddSquares(sum2, *reinterpret_cast<const float4 *>(&sm.F[s][x]));
        }
        float discr, mult;
        NormScales(sum2, 128, &discr, &mult);
        sm.Mult[s] = mult;
    }
    __syncthreads();
    QuantiseStaged(p, sm, 0, 32, false);
}

// The contract product's input: relu of the expand sums normalised per head (groups of ReluDim / Heads columns).  A group that lies
// inside the chunk is summed from shared memory, one that reaches beyond it from L2.
__device__ __forceinline__ void NormaliseRelu(const TStepParams &p, TStepSmem &sm, int chunk)
{
    // three loads of a thread before the first use (an unrolled loop ran its five or six iterations in the remainder, one load after the
    // other)
#pragma unroll 1
    for (int base = threadIdx.x; base < p.NSeq * 32; base += PS_STAGE_AHEAD * PS_THREADS) {
        int4 a[PS_STAGE_AHEAD];
#pragma unroll
        for (int k = 0; k < PS_STAGE_AHEAD; ++k) {
            const int i = base + k * PS_THREADS;
            if (i < p.NSeq * 32) {
                a[k] = __ldcg(reinterpret_cast<const int4 *>(p.Expand + (size_t)(i >> 5) * p.ReluDim + chunk * 128 + (i & 31) * 4));
            }
        }
#pragma unroll
        for (int k = 0; k < PS_STAGE_AHEAD; ++k) {
            const int i = base + k * PS_THREADS;
            if (i < p.NSeq * 32) {
                *reinterpret_cast<float4 *>(&sm.F[i >> 5][(i & 31) * 4]) = make_float4((float)a[k].x, (float)a[k].y, (float)a[k].z, (float)a[k].w);
            }
        }
    }
    __syncthreads();
    const int group = p.ReluDim / p.Heads, c0 = chunk * 128;
    if (group % 16 != 0) {
        // head sizes no model of the family has: a thread per 16 columns adds up the groups they belong to by itself
        for (int i = threadIdx.x; i < p.NSeq * 8; i += PS_THREADS) {
            const int s = i >> 3, c16 = i & 7;
            const int *src = p.Expand + (size_t)s * p.ReluDim;
            uint32_t w[4] = {0, 0, 0, 0};
            int cur = -1;
            float mult = 0;
            for (int k = 0; k < 16; ++k) {
                const int col = c0 + c16 * 16 + k;
                if (col / group != cur) {
                    cur = col / group;
                    float sum2 = 0, discr;
                    for (int x = cur * group; x < (cur + 1) * group; ++x) {
                        const float a = (float)__ldcg(src + x);
                        sum2 = __fadd_rn(sum2, __fmul_rn(a, a));
                    }
                    NormScales(sum2, group, &discr, &mult);
                }
                w[k >> 2] |= (uint32_t)(max(ToInt8Clamp127(__fmul_rn(sm.F[s][c16 * 16 + k], mult)), 0) & 0xff) << (8 * (k & 3));
            }
            StoreCodes(sm.B, s, c16, make_int4((int)w[0], (int)w[1], (int)w[2], (int)w[3]));
        }
        return;
    }
    for (int g = c0 / group; g * group < c0 + 128; ++g) {
        const int g0 = g * group, g1 = g0 + group;
        const int s = threadIdx.x;
        if (s < p.NSeq) {
            float sum2 = 0;
            if (g0 >= c0 && g1 <= c0 + 128) {
#pragma unroll 8
                for (int x = g0 - c0; x < g1 - c0; x += 4) {
                    sum2 = AddSquares(sum2, *reinterpret_cast<const float4 *>(&sm.F[s][x]));
                }
            } else {
                const int4 *src = reinterpret_cast<const int4 *>(p.Expand + (size_t)s * p.ReluDim + g0);
#pragma unroll 8
                for (int x = 0; x < group / 4; ++x) {
                    const int4 a = __ldcg(src + x);
                    sum2 = AddSquares(sum2, make_float4((float)a.x, (float)a.y, (float)a.z, (float)a.w));
                }
            }
            float discr, mult;
            NormScales(sum2, group, &discr, &mult);
            sm.Mult[s] = mult;
        }
        __syncthreads();
        const int lo = max(g0, c0) - c0, hi = min(g1, c0 + 128) - c0;
        QuantiseStaged(p, sm, lo / 4, (hi - lo) / 4, true);
        if (g1 < c0 + 128) {
            __syncthreads(); // the next group overwrites sm.Mult
        }
    }
}

// All of this CTA's items of one matrix product.
__device__ __forceinline__ void ProductPhase(const TStepParams &p, TStepSmem &sm, int l, int phase, TTileCursor &cursor)
{
    const int tid = threadIdx.x, warp = tid >> 5;
    const int hs = p.Heads * p.HeadSize;
    const int nCols = (p.NSeq + 15) & ~15; // accumulator columns
    const uint32_t idesc = MakeInstrDesc(2, 1, 1, 0, 0, 128, nCols);
    const int end = sm.PhaseBegin[phase + 1];
    for (int index = sm.PhaseBegin[phase]; index < end; ++index) {
        const TWeightTile t = TileAt(p, sm, index);
        const int chunk = t.Chunk, tile = t.Matrix == 0 || t.Matrix > 3 ? t.Tile : -1; // tile 0 of the phase also keeps the new state
        if (phase == PH_PROJ || phase == PH_EXPAND) {
            // StateA and StateB take turns: the first holds the state in front of the attention block, the second behind it
            const bool proj = phase == PH_PROJ;
            const int source = proj && l == 0 ? p.FirstSource : SRC_SUM;
            StageState(p, sm, chunk, source, proj == (source == SRC_SUM) ? p.StateB : p.StateA, proj ? p.Contract : p.Comb,
                proj ? sm.Now.PrevContractScale : sm.Now.CombScale, tile != 0 || source == SRC_STATE ? nullptr : proj ? p.StateA : p.StateB);
            NormaliseStaged(p, sm);
        } else if (phase == PH_COMB) {
#pragma unroll 2
            for (int i = tid; i < p.NSeq * 8; i += PS_THREADS) {
                StoreCodes(sm.B, i >> 3, i & 7, __ldcg(reinterpret_cast<const int4 *>(p.Kv8 + (size_t)(i >> 3) * 4 * hs + chunk * 128 + (i & 7) * 16)));
            }
        } else {
            NormaliseRelu(p, sm, chunk);
        }
        // this thread's part of the tile has landed: the groups requested behind it (one per tile, at most PS_RING - 1 tiles are
        // requested and not used up) may still be on their way
        if (cursor.Requested - cursor.Used == PS_RING - 1) {
            CpAsyncWait<PS_RING - 2>();
        } else {
            CpAsyncWait<0>();
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        TcFenceBefore();
        __syncthreads();
        TcFenceAfter();
        if (warp == 0 && ElectOne()) {
            const uint32_t sA = SmemAddr(sm.Ring[cursor.Used % PS_RING]), sB = SmemAddr(sm.B);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
                MmaI8SS(sm.TmemBase, MakeSmemDesc(sA + ks * 32, 16, 1024, 128), MakeSmemDesc(sB + ks * 32, 16, 1024, 128), idesc,
                    (!(t.Flags & TILE_FIRST) || ks > 0) ? 1u : 0u);
            }
            MmaCommit(&sm.MmaDone);
        }
        if (!WaitBar(&sm.MmaDone, cursor.Used & 1)) {
            sm.Failed = 1;
            if (p.Status) {
                atomicOr(p.Status, kDevTimeoutMma);
            }
        }
        ++cursor.Used;
        if (cursor.Requested - cursor.Used < PS_RING / 2) {
            RefillRing(p, sm, &cursor); // a phase with many tiles for one CTA: do not wait for its end
        }
        if (!(t.Flags & TILE_LAST)) {
            continue;
        }
        TcFenceAfter();
        // 128 rows x 16 sequences per warp: the item's sums join the others' in L2.  Written as sixteen predicated additions they were
        // a kilobyte of instructions that every phase fetched anew, for one sequence too (1 K of the 7 K clocks of a phase)
        int *out = phase == PH_PROJ ? p.Proj + t.Matrix * hs : phase == PH_COMB ? p.Comb : phase == PH_EXPAND ? p.Expand : p.Contract;
        const int rows = phase == PH_PROJ ? hs : phase == PH_EXPAND ? p.ReluDim : p.Dim, pitch = phase == PH_PROJ ? 4 * hs : rows;
        const int quad = warp & 3, row = t.Tile * 128 + quad * 32 + (tid & 31);
        for (int s0 = (warp >> 2) * 16; s0 < nCols; s0 += PS_GROUPS * 16) {
            uint32_t acc[16];
            TmemLd16(sm.TmemBase + ((uint32_t)(quad * 32) << 16) + s0, acc);
            TmemWaitLd();
            if (row < rows) {
                int *dst = out + (size_t)s0 * pitch + row;
#pragma unroll
                for (int j = 0; j < 16; j += 4) {
                    if (s0 + j >= p.NSeq) { // the rest has no sequences: nor its instructions to be fetched
                        break;
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        if (s0 + j + k < p.NSeq) {
                            atomicAdd(dst, (int)acc[j + k]);
                        }
                        dst += pitch;
                    }
                }
            }
        }
        TcFenceBefore();
        if (index + 1 < end) {
            __syncthreads(); // the accumulators have been read
        }
    }
}

// ---- attention -----------------------------------------------------------------------------------------------------
// Every sequence's keys are cut into chunks of one size, counted from the first key it attends: the smallest multiple of eight (at
// least PS_MIN_CHUNK) that gives no more than PS_CHUNKS_PER_SM chunks per SM, the rule of the decode kernel (DecodePlan), and a
// chunk into Split parts of whole batches of eight.  Sums are formed in that order and no other: keys of a part one batch after
// another, parts of a chunk, chunks of a row.  So the bits of a sequence's result depend on the chunk size alone, not on its slot or
// on which unit takes what, and are those of the decode kernel's chunks merged one after another.
// A warp-wide 16-byte load covers a head group (AttGroupHeads) for one stream of keys or several; a stream is one part of one
// chunk.  A unit = as many consecutive chunks as four warps have streams for x one head group, taken by a group of four warps.
// Its chunks may belong to several sequences.
__device__ __forceinline__ bool PosOk(const TStepParams &p, int pos)
{
    return pos >= 0 && pos < p.RopeLen && pos < p.Capacity;
}

// by one warp, into shared memory; pos: lane i has those of sequences i and i + 32
__device__ __noinline__ void MakeAttPlan(const TStepParams &p, int window, int pos0, int pos1, TAttPlan &plan)
{
    const int lane = threadIdx.x & 31;
    auto keysOf = [&](int s, int pos) {
        int j0 = 0, j1 = 0;
        if (s < p.NSeq && PosOk(p, pos)) {
            KeyRange(pos + 1, window, &j0, &j1);
        }
        return j1 - j0;
    };
    auto warpSum = [](int v) { return (int)__reduce_add_sync(0xffffffffu, (unsigned)v); };
    const int k0 = keysOf(lane, pos0), k1 = keysOf(lane + 32, pos1);
    const int total = warpSum(k0 + k1), target = min((int)gridDim.x * PS_CHUNKS_PER_SM, INF_MAX_CHUNKS);
    int chunk = max(((total + target - 1) / target + 7) & ~7, PS_MIN_CHUNK);
    if (p.NSeq < target) {
        // a sequence's last chunk is a partial one: the count falls as the size grows, total / (target - NSeq) is always enough
        int lo = chunk / 8, hi = max(((total + (target - p.NSeq) - 1) / (target - p.NSeq) + 7) / 8, lo);
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (warpSum((k0 + mid * 8 - 1) / (mid * 8) + (k1 + mid * 8 - 1) / (mid * 8)) <= target) {
                hi = mid;
            } else {
                lo = mid + 1;
            }
        }
        chunk = lo * 8;
    }
    // a sequence without keys has a chunk too: the unit that takes it appends the new token
    const int n0 = lane < p.NSeq ? max((k0 + chunk - 1) / chunk, 1) : 0, n1 = lane + 32 < p.NSeq ? max((k1 + chunk - 1) / chunk, 1) : 0;
    const int parts = min(p.Split, chunk / 8), perUnit = (4 << p.PerLoadLog) / parts; // no part is shorter than a batch
    // every sequence begins with a unit of its own where the groups of four warps suffice for that: rows that fit a unit then need no
    // partials
    const int w0 = (n0 + perUnit - 1) / perUnit, w1 = (n1 + perUnit - 1) / perUnit, whole = warpSum(w0 + w1);
    const bool apart = whole * p.HeadGroups <= (int)gridDim.x * PS_GROUPS && whole * perUnit <= INF_MAX_CHUNKS;
    const int t0 = apart ? w0 * perUnit : n0, t1 = apart ? w1 * perUnit : n1;
    int i0 = t0, i1 = t1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, i0, o), b = __shfl_up_sync(0xffffffffu, i1, o);
        i0 += lane >= o ? a : 0;
        i1 += lane >= o ? b : 0;
    }
    const int sum0 = __shfl_sync(0xffffffffu, i0, 31), slots = sum0 + __shfl_sync(0xffffffffu, i1, 31);
    const int b0 = i0 - t0, b1 = sum0 + i1 - t1;
    plan.Pos[lane] = pos0;
    plan.Pos[lane + 32] = pos1;
    plan.Base[lane] = b0;
    plan.Base[lane + 32] = b1;
    plan.Count[lane] = n0;
    plan.Count[lane + 32] = n1;
    for (int i = 0; i < t0; ++i) {
        plan.SeqOf[b0 + i] = (uint8_t)lane;
    }
    for (int i = 0; i < t1; ++i) {
        plan.SeqOf[b1 + i] = (uint8_t)(lane + 32);
    }
    if (lane == 0) {
        plan.Window = window;
        plan.Chunk = chunk;
        plan.Parts = parts;
        plan.PerUnit = perUnit;
        plan.Slots = slots;
        // neighbouring units, the head groups of the same chunks, on one SM
        const long long units = (slots + perUnit - 1) / perUnit * p.HeadGroups;
        plan.UnitBegin = (int)(units * blockIdx.x / gridDim.x);
        plan.UnitEnd = (int)(units * (blockIdx.x + 1) / gridDim.x);
    }
    __syncwarp();
}

// What the attention of layer l needs besides the projections, while the CTA waits for them: the plan (warp 1; the one in shared
// memory if window and positions are the same) and the table of the caches (warps 2 and 3).
__device__ __noinline__ void PrepareAttention(const TStepParams &p, TStepSmem &sm, int l)
{
    const TStepLayer &layer = p.Layers[l];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp == 1) {
        const int pos0 = lane < p.NSeq ? layer.CtxLens[lane] : 0, pos1 = lane + 32 < p.NSeq ? layer.CtxLens[lane + 32] : 0;
        auto report = [&](int s, int pos) {
            if (s < p.NSeq && (!PosOk(p, pos) || pos + 1 > p.MaxCtx) && p.Status) {
                atomicOr(p.Status, kDevBadSpan); // the cache or the rope table is full, or longer than the caller's bound
            }
        };
        if (blockIdx.x == 0) {
            report(lane, pos0);
            report(lane + 32, pos1);
        }
        int slot = -1;
        for (int i = 0; i < 2; ++i) {
            const TAttPlan &plan = sm.Plan[i];
            if (plan.Window == layer.Window && __all_sync(0xffffffffu, plan.Pos[lane] == pos0 && plan.Pos[lane + 32] == pos1)) {
                slot = i;
            }
        }
        if (slot < 0) {
            slot = sm.Plan[0].Window < 0 ? 0 : sm.Plan[1].Window < 0 ? 1 : sm.PlanOf ^ 1; // the one not used last
            __syncwarp();
            MakeAttPlan(p, layer.Window, pos0, pos1, sm.Plan[slot]);
        }
        if (lane == 0) {
            sm.PlanOf = slot;
        }
    } else if (warp == 2 || warp == 3) {
        const int s = (int)threadIdx.x - 64;
        if (s < p.NSeq) {
            sm.Seqs[s] = layer.Seqs[s];
        }
    }
}

// The combiner input of four consecutive columns z .. z + 3 of a head: kv[blk][z] = int8(key[z ^ blk] * val[z]) (KVProduct,
// cpu_infer.cpp:318-337); z ^ blk stays among the four.
__device__ __forceinline__ void StoreKvProduct(int8_t *kv, int headSize, int z, char4 key, const float *val)
{
    const int k[4] = {key.x, key.y, key.z, key.w};
#pragma unroll
    for (int blk = 0; blk < 4; ++blk) {
        uint32_t w = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            w |= (uint32_t)(ToInt8Clamp127(__fmul_rn((float)k[i ^ blk], val[i])) & 0xff) << (8 * i);
        }
        *reinterpret_cast<uint32_t *>(kv + blk * headSize + z) = w;
    }
}

// One matrix (m: qk, qv, k, v) of a head group of one sequence, by one warp: rope on qk and qv (ReferenceApplyRope,
// code/gpt/att/rope.cpp:28-46), NormalizeState per head, codes into shared memory (qk, k: at `codes`) or the sequence's cache (qv, v).
template <int D>
__device__ __noinline__ void ProjectHeads(const TStepParams &p, float qvMult, TAttGroupSmem &g, const tsa_kv_seq &sq, int m, int seq, int codes,
    int head0, int heads, int pos)
{
    const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) & 3, hs = p.Heads * D;
    const int *src = p.Proj + (size_t)seq * 4 * hs + m * hs + head0 * D;
    float *rot = g.Rot[warp];
    // up to eight blocks of 64 columns, all loads in flight at once
    constexpr int PER_HEAD = D / 64;
    const int blocks = heads * PER_HEAD;
    float cs[PER_HEAD], sn[PER_HEAD];
    int v0[8], v1[8];
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        if (b < blocks) {
            v0[b] = __ldcg(src + b * 64 + lane);
            v1[b] = __ldcg(src + b * 64 + lane + 32);
        }
    }
    if (m < 2) {
        const float *rp = p.Rope + (size_t)pos * D;
#pragma unroll
        for (int b = 0; b < PER_HEAD; ++b) {
            cs[b] = __ldg(rp + b * 64 + lane);
            sn[b] = __ldg(rp + b * 64 + lane + 32);
        }
    }
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        if (b < blocks) {
            float r0 = (float)v0[b], r1 = (float)v1[b];
            if (m < 2) {
                const float x0 = r0, x1 = r1, c = cs[b % PER_HEAD], s = sn[b % PER_HEAD];
                r0 = __fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, s));
                r1 = __fadd_rn(__fmul_rn(x0, s), __fmul_rn(x1, c));
            }
            float *w = rot + (b / PER_HEAD) * (D + 4) + (b % PER_HEAD) * 64;
            w[lane] = r0;
            w[lane + 32] = r1;
        }
    }
    __syncwarp();
    if (lane < heads) {
        const float *w = rot + lane * (D + 4);
        float sum2 = 0;
#pragma unroll 16
        for (int x = 0; x < D; x += 4) {
            sum2 = AddSquares(sum2, *reinterpret_cast<const float4 *>(w + x));
        }
        float discr, mult;
        NormScales(sum2, D, &discr, &mult);
        g.Mult[warp][lane] = mult;
        if (m == 1) {
            ((float *)sq.kScale)[(size_t)pos * p.Heads + head0 + lane] = __fmul_rn(discr, qvMult);
        } else if (m == 3) {
            ((float *)sq.vScale)[(size_t)pos * p.Heads + head0 + lane] = INF_VEC_SCALE;
        }
    }
    __syncwarp();
    // four columns per lane and step
    for (int i = lane * 4; i < heads * D; i += 128) {
        const int h = i / D;
        const float4 w = *reinterpret_cast<const float4 *>(rot + h * (D + 4) + (i & (D - 1)));
        const float mult = g.Mult[warp][h];
        char4 q;
        q.x = (char)ToInt8Clamp127(__fmul_rn(w.x, mult));
        q.y = (char)ToInt8Clamp127(__fmul_rn(w.y, mult));
        q.z = (char)ToInt8Clamp127(__fmul_rn(w.z, mult));
        q.w = (char)ToInt8Clamp127(__fmul_rn(w.w, mult));
        if (m == 0) {
            *reinterpret_cast<char4 *>(g.Q8 + codes + i) = q;
        } else if (m == 2) {
            *reinterpret_cast<char4 *>(g.K8 + codes + i) = q;
            *reinterpret_cast<char4 *>(p.K8 + (size_t)seq * hs + head0 * D + i) = q;
        } else {
            *reinterpret_cast<char4 *>((int8_t *)(m == 1 ? sq.k : sq.v) + (size_t)pos * hs + head0 * D + i) = q;
        }
    }
    __syncwarp(); // the warp's buffers are used again for its next matrix
}

// four columns of a row's result, times the combiner key (its codes in shared memory, or null: in L2), as codes for the combiner
template <int D>
__device__ __noinline__ void FinishColumns(const TStepParams &p, int pos, int seq, int head, int z, const int8_t *keyCodes, float sum, float4 acc)
{
    const size_t row = (size_t)seq * p.Heads * D;
    char4 key = make_char4(0, 0, 0, 0);
    float val[4] = {0, 0, 0, 0};
    if (PosOk(p, pos)) {
        const int packed = keyCodes ? *reinterpret_cast<const int *>(keyCodes) : __ldcg(reinterpret_cast<const int *>(p.K8 + row + head * D + z));
        key = *reinterpret_cast<const char4 *>(&packed);
        val[0] = acc.x / sum, val[1] = acc.y / sum, val[2] = acc.z / sum, val[3] = acc.w / sum;
    }
    StoreKvProduct(p.Kv8 + (row + head * D) * 4, D, z, key, val);
}

// all chunks of a row, their partials one step of all heads apart, and the sink
template <int D>
__device__ __noinline__ void MergePartials(const TStepParams &p, const float *src, int chunks, int z, float &sum, float (&val)[4])
{
    const size_t step = (size_t)p.Heads * (D + 4);
    constexpr int LPH = D / 16;
    float mAll = 0; // the sink has logit 0 (softMax.Add(0), cpu_infer.cpp:444)
#pragma unroll 4
    for (int c = (threadIdx.x & 31) % LPH; c < chunks; c += LPH) { // shared out among the lanes of the head
        mAll = fmaxf(mAll, __ldcg(src + c * step + D));
    }
#pragma unroll
    for (int o = LPH / 2; o > 0; o >>= 1) {
        mAll = fmaxf(mAll, __shfl_xor_sync(0xffffffffu, mAll, o));
    }
    float sumAll = exp2f(-mAll);
    float4 acc = make_float4(0, 0, 0, 0);
#pragma unroll 4
    for (int c = 0; c < chunks; ++c) {
        const float2 ml = __ldcg(reinterpret_cast<const float2 *>(src + c * step + D));
        const float4 v = __ldcg(reinterpret_cast<const float4 *>(src + c * step + z));
        const float f = exp2f(ml.x - mAll);
        sumAll = fmaf(f, ml.y, sumAll);
        acc.x = fmaf(f, v.x, acc.x);
        acc.y = fmaf(f, v.y, acc.y);
        acc.z = fmaf(f, v.z, acc.z);
        acc.w = fmaf(f, v.w, acc.w);
    }
    sum = sumAll;
    val[0] = acc.x, val[1] = acc.y, val[2] = acc.z, val[3] = acc.w;
}

// this lane's stream of keys, its maximum, sum and columns into the merge buffer
template <int D>
__device__ __forceinline__ void AttendRange(const int4 qv, float logitMult, float slope, int pos, const int8_t *k, const int8_t *v, const float *ks, const float *vs,
    int heads, int tBeg, int tEnd, int batches, float *mine)
{
    float m = -1e30f, sum = 0, acc[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        acc[i] = 0;
    }
    AttendTokens<D, 8, true>(qv, logitMult, slope, pos, reinterpret_cast<const int4 *>(k), reinterpret_cast<const int4 *>(v), ks, vs, heads, tBeg, tEnd, batches, m,
        sum, acc);
    const bool any = tBeg < tEnd;
    mine[0] = m;
    mine[1] = any ? sum : 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        mine[2 + i] = any ? acc[i] : 0.0f;
    }
}

template <int D>
__device__ void AttentionPhase(const TStepParams &p, TStepSmem &sm)
{
    constexpr int LPH = D / 16;  // lanes per head
    constexpr int PITCH = D + 4; // of a partial: columns, maximum, sum
    const TAttPlan &plan = sm.Plan[sm.PlanOf];
    const int tid = threadIdx.x, lane = tid & 31, group = tid >> 7, w = (tid >> 5) & 3;
    const int hs = p.Heads * D;
    TAttGroupSmem &g = sm.Att[group];
    // this lane's stream among those of a load, head inside the group, 16-byte slice of the head; lanes past the last stream repeat the first's
    const int streamLanes = p.PerGroup * LPH, perLoad = 1 << p.PerLoadLog;
    const int streamOff = lane / streamLanes < perLoad ? lane / streamLanes : 0, first = lane % streamLanes;
    const int head = first / LPH, sub = lane % LPH, z = sub * 16 + 4 * w;
    for (int unit = plan.UnitBegin + group; unit < plan.UnitEnd; unit += PS_GROUPS) {
        const int range = unit / p.HeadGroups, hg = unit - range * p.HeadGroups, head0 = hg * p.PerGroup, heads = min(p.PerGroup, p.Heads - head0);
        const int slot0 = range * plan.PerUnit, slots = min(plan.PerUnit, plan.Slots - slot0);
        const int seq0 = plan.SeqOf[slot0], seq1 = plan.SeqOf[slot0 + slots - 1];
        // the four matrices of a sequence by the four warps; only the unit with its first chunk appends the token and leaves the combiner key
        for (int seq = seq0; seq <= seq1; ++seq) {
            const int m = (w + seq - seq0) & 3, pos = plan.Pos[seq];
            if (PosOk(p, pos) && (m == 0 || plan.Base[seq] >= slot0)) {
                ProjectHeads<D>(p, sm.Now.QvMult, g, sm.Seqs[seq], m, seq, (seq - seq0) * p.PerGroup * D, head0, heads, pos);
            }
        }
        GroupSync(group);
        {
            // this lane's stream: part `part` of chunk `chunk` of the unit
            const int stream = (w << p.PerLoadLog) + streamOff, parts = plan.Parts;
            const int chunk = parts == 3 ? stream / 3 : stream >> (parts >> 1), part = stream - chunk * parts;
            int tBeg = 1, tEnd = 1, seq = seq0; // none: the lane reads the first key and takes nothing from it
            if (chunk < slots) {
                seq = plan.SeqOf[slot0 + chunk];
                int j0, j1;
                KeyRange(plan.Pos[seq] + 1, sm.Now.Window, &j0, &j1);
                const int cBeg = j0 + (slot0 + chunk - plan.Base[seq]) * plan.Chunk, cEnd = min(cBeg + plan.Chunk, j1);
                const int perPart = (((cEnd - cBeg + p.Split - 1) >> (p.Split >> 1)) + 7) & ~7, beg = cBeg + part * perPart, end = min(beg + perPart, cEnd);
                if (beg < end && PosOk(p, plan.Pos[seq])) {
                    tBeg = beg;
                    tEnd = end;
                }
            }
            const int batches = __reduce_max_sync(0xffffffffu, (unsigned)(tEnd - tBeg + 7) / 8);
            const int headC = head0 + min(head, heads - 1);
            const tsa_kv_seq &sq = sm.Seqs[seq];
            const int4 qv = *reinterpret_cast<const int4 *>(g.Q8 + (seq - seq0) * p.PerGroup * D + (headC - head0) * D + sub * 16);
            const size_t off = (size_t)tBeg * hs + headC * D + sub * 16, soff = (size_t)tBeg * p.Heads + headC;
            AttendRange<D>(qv, p.DotScale * INF_VEC_SCALE, sm.Now.Slope, plan.Pos[seq], (const int8_t *)sq.k + off, (const int8_t *)sq.v + off,
                (const float *)sq.kScale + soff, (const float *)sq.vScale + soff, p.Heads, tBeg, tEnd, batches, g.Merge[w][lane]);
        }
        GroupSync(group);
        // Warp w goes on with columns 4 w .. 4 w + 3 of every slice.
        auto shareOf = [&](int stream) { return (const float *)g.Merge[stream >> p.PerLoadLog][first + (stream & (perLoad - 1)) * streamLanes]; };
        // the parts of a chunk
        auto mergeChunk = [&](int chunk, float &m, float &sum, float (&val)[4]) {
            const float *share = shareOf(chunk * plan.Parts);
            m = share[0];
            sum = share[1];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                val[i] = share[2 + 4 * w + i];
            }
            for (int k = 1; k < plan.Parts; ++k) {
                const float *other = shareOf(chunk * plan.Parts + k);
                const float mAll = fmaxf(m, other[0]);
                const float c1 = exp2f(m - mAll), c2 = exp2f(other[0] - mAll);
                sum = sum * c1 + other[1] * c2;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    val[i] = val[i] * c1 + other[2 + 4 * w + i] * c2;
                }
                m = mAll;
            }
        };
        auto finish = [&](int seq, float sum, const float (&val)[4]) {
            if (head < heads && lane < streamLanes) {
                const int8_t *key = plan.Base[seq] >= slot0 ? g.K8 + (seq - seq0) * p.PerGroup * D + head * D + z : nullptr;
                FinishColumns<D>(p, plan.Pos[seq], seq, head0 + head, z, key, sum, make_float4(val[0], val[1], val[2], val[3]));
            }
        };
        auto chunksHere = [&](int seq, int &c0, int &c1) { // the unit's chunks of a sequence
            c0 = max(plan.Base[seq] - slot0, 0);
            c1 = min(plan.Base[seq] + plan.Count[seq] - slot0, slots);
            return c1 - c0;
        };
        bool shared = false; // a row that other units have chunks of: its partials go to L2
        for (int seq = seq0; seq <= seq1; ++seq) {
            int c0, c1;
            const bool whole = chunksHere(seq, c0, c1) == plan.Count[seq];
            shared |= !whole;
            float mAll = 0; // the sink has logit 0 (softMax.Add(0), cpu_infer.cpp:444)
            if (whole) {
                for (int k = c0 * plan.Parts; k < c1 * plan.Parts; ++k) {
                    mAll = fmaxf(mAll, shareOf(k)[0]);
                }
            }
            float sumAll = exp2f(-mAll), valAll[4] = {0, 0, 0, 0};
            for (int c = c0; c < c1; ++c) {
                float m, sum, val[4];
                mergeChunk(c, m, sum, val);
                if (whole) {
                    const float f = exp2f(m - mAll);
                    sumAll = fmaf(f, sum, sumAll);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        valAll[i] = fmaf(f, val[i], valAll[i]);
                    }
                } else if (head < heads && lane < streamLanes) {
                    float *dst = p.Partial + ((size_t)(slot0 + c) * p.Heads + head0 + head) * PITCH;
                    __stcg(reinterpret_cast<float4 *>(dst + z), make_float4(val[0], val[1], val[2], val[3]));
                    if (z == 0) {
                        __stcg(reinterpret_cast<float2 *>(dst + D), make_float2(m, sum));
                    }
                }
            }
            if (whole) {
                finish(seq, sumAll, valAll);
            }
        }
        if (shared) {
            // at most the first and the last sequence; the unit that arrives last merges all chunks of the row
            GroupSync(group);
            if (tid % 128 < 2) {
                const int seq = tid % 128 == 0 ? seq0 : seq1;
                int c0, c1, last = 0;
                const int here = chunksHere(seq, c0, c1);
                if (here != plan.Count[seq] && (tid % 128 == 0 || seq1 != seq0)) {
                    int *arrived = p.Arrived + seq * p.HeadGroups + hg;
                    int before;
                    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], %2;" : "=r"(before) : "l"(arrived), "r"(here) : "memory");
                    last = before + here == plan.Count[seq];
                    if (last) {
                        *arrived = 0; // for the next layer
                    }
                }
                g.Last[tid % 128] = last;
            }
            GroupSync(group);
            for (int k = 0; k < 2; ++k) {
                if (!g.Last[k]) {
                    continue;
                }
                const int seq = k == 0 ? seq0 : seq1, chunks = plan.Count[seq];
                float sumAll, valAll[4];
                MergePartials<D>(p, p.Partial + ((size_t)plan.Base[seq] * p.Heads + head0 + min(head, heads - 1)) * PITCH, chunks, z, sumAll, valAll);
                finish(seq, sumAll, valAll);
            }
        }
        GroupSync(group); // the group's shared memory is used again by its next unit
    }
}

__device__ __forceinline__ void ZeroSums(int *sums, int n)
{
    for (int i = blockIdx.x * PS_THREADS + threadIdx.x; i < n / 4; i += gridDim.x * PS_THREADS) {
        reinterpret_cast<int4 *>(sums)[i] = make_int4(0, 0, 0, 0);
    }
}

__device__ __forceinline__ TLayerNow LayerNow(const TStepParams &p, int l)
{
    TLayerNow n;
    n.QvMult = p.Layers[l].QvMult;
    n.CombScale = p.Layers[l].CombScale;
    n.PrevContractScale = l > 0 ? p.Layers[l - 1].ContractScale : 0.0f;
    n.Slope = p.Layers[l].Slope;
    n.Window = p.Layers[l].Window;
    return n;
}

template <int D>
__device__ void RunLayers(const TStepParams &p, TStepSmem &sm)
{
    const int tid = threadIdx.x, hs = p.Heads * D;
    if (tid < 5) {
        int n = 0;
        for (int phase = 0; phase < tid; ++phase) {
            const TStepShape &s = p.Shape[phase];
            for (int item = blockIdx.x; item < s.Tiles * s.Splits; item += gridDim.x) {
                n += min(s.Per, s.Chunks - (item % s.Splits) * s.Per);
            }
        }
        sm.PhaseBegin[tid] = n;
    }
    if (tid == PS_THREADS - 1 && p.LayerCount > 0) {
        sm.Now = LayerNow(p, 0);
    }
    __syncthreads();
    for (int i = tid; i < sm.PhaseBegin[4] && i < PS_TABLE; i += PS_THREADS) {
        sm.Table[i] = ComputeTile(p, i);
    }
    __syncthreads();
    TTileCursor cursor = {0, 0, sm.PhaseBegin[4] > 0 ? 0 : p.LayerCount, 0};
    RefillRing(p, sm, &cursor);
    // One loop over all phases, so that every piece of code exists once: the kernel's loop has to fit the SM's instruction cache
    // (with the phases written out one after another a quarter of the instruction fetches missed it).
    // Sums are cleared a phase or more after their last reader has passed a barrier and a phase or more before their next writer.
    int l = 0, phase = PH_PROJ;
    bool attention = false; // the attention follows PH_PROJ
#pragma unroll 1
    while (l < p.LayerCount) {
        if (attention) {
            ZeroSums(l > 0 ? p.Contract : p.Comb, p.NSeq * p.Dim);
            AttentionPhase<D>(p, sm);
        } else {
            int *done = phase == PH_PROJ ? p.Expand : phase == PH_COMB ? p.Proj : p.Comb;
            const int doneInts = p.NSeq * (phase == PH_PROJ ? p.ReluDim : phase == PH_COMB ? 4 * hs : p.Dim);
            if (phase != PH_EXPAND && (phase != PH_PROJ || l > 0)) {
                ZeroSums(done, doneInts);
            }
            if (phase == PH_COMB && blockIdx.x == gridDim.x - 1 && tid < p.NSeq) {
                p.Layers[l].CtxLens[tid] += 1; // the token is in every sequence's cache of this layer
            }
            ProductPhase(p, sm, l, phase, cursor);
        }
        GridArrive(p);
        if (!attention && phase == PH_PROJ) {
            PrepareAttention(p, sm, l);
        }
        if (!attention && phase == PH_CONTRACT && tid == PS_THREADS - 1 && l + 1 < p.LayerCount) {
            sm.Now = LayerNow(p, l + 1);
        }
        RefillRing(p, sm, &cursor);
        if (!attention && phase == PH_PROJ) {
            attention = true;
        } else {
            attention = false;
            if (++phase == 4) {
                phase = PH_PROJ;
                ++l;
            }
        }
        if (!GridWait(p, sm)) {
            return;
        }
    }
    // the state after the last layer: fp32 for a launch that continues from here, its int8 form for the final product
    for (int chunk = blockIdx.x; chunk < p.Dim / 128; chunk += gridDim.x) {
        StageState(p, sm, chunk, p.LayerCount > 0 ? SRC_SUM : p.FirstSource, p.StateB, p.Contract, p.LayerCount > 0 ? p.Layers[p.LayerCount - 1].ContractScale : 0.0f,
            p.StateA);
        NormaliseStaged(p, sm);
        __syncthreads();
        for (int i = tid; i < p.NSeq * 8; i += PS_THREADS) {
            const int s = i >> 3, c16 = i & 7;
            *reinterpret_cast<int4 *>(p.NormState + (size_t)s * p.Dim + chunk * 128 + c16 * 16) = *reinterpret_cast<const int4 *>(sm.B + s * 128 + ((c16 ^ (s & 7)) << 4));
        }
        __syncthreads();
    }
}

// PS_THREADS x 168 registers and nearly all of the shared memory: one CTA per SM.
template <int D>
__global__ void __launch_bounds__(PS_THREADS, 1) InferLayersKernel(const __grid_constant__ TStepParams p)
{
    extern __shared__ uint8_t stepSmemRaw[];
    TStepSmem &sm = *reinterpret_cast<TStepSmem *>(((uintptr_t)stepSmemRaw + 1023) & ~(uintptr_t)1023); // operand tiles: 128-byte swizzle
    const int tid = threadIdx.x;
    PdlWait();
    if (tid == 0) {
        MbarInit(&sm.MmaDone, 1);
        FenceBarrierInit();
        sm.Failed = 0;
        sm.Passed = 0;
        sm.Plan[0].Window = sm.Plan[1].Window = -1;
        sm.PlanOf = 0;
    }
    if (tid < 32) {
        TmemAlloc(&sm.TmemBase, 64);
        TmemRelinquish();
    }
    for (int i = tid; i < PS_B_BYTES / 16; i += PS_THREADS) {
        reinterpret_cast<int4 *>(sm.B)[i] = make_int4(0, 0, 0, 0); // rows past the batch stay zero
    }
    TcFenceBefore();
    __syncthreads();
    TcFenceAfter();
    RunLayers<D>(p, sm);
    CpAsyncWait<0>();
    TcFenceBefore();
    __syncthreads();
    PdlTrigger();
    if (tid < 32) {
        TmemDealloc(sm.TmemBase, 64);
    }
}

int InferLayersPersistent(const tsa_infer_model *model, const tsa_kv_seq *const *layerSeqs, int *ctxLens, int capacity, const int *labels, int labelsPerSeq,
    int nSeq, int maxCtx, const TInferBuffers &b, int *statusWord, cudaStream_t stream)
{
    const tsa_infer_dims &d = model->dims;
    const int hs = d.head_count * d.head_dim, D = d.head_dim;
    int dev = 0, sms = 0;
    int rc = CheckCuda(cudaGetDevice(&dev), "cudaGetDevice");
    if (rc == TSA_OK) {
        rc = CheckCuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "cudaDeviceGetAttribute");
    }
    const void *kern = D == 64 ? (const void *)InferLayersKernel<64> : (const void *)InferLayersKernel<128>;
    const int smemBytes = (int)sizeof(TStepSmem) + 1024;
    if (rc == TSA_OK) {
        rc = CheckCuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smemBytes), "cudaFuncSetAttribute(inference layers)");
    }
    if (rc != TSA_OK) {
        return rc;
    }
    TStepParams p;
    auto shape = [&](int tiles, int columns) {
        // as many items as SMs, each with the same number of column chunks
        TStepShape s;
        s.Tiles = tiles;
        s.Chunks = columns / 128;
        int splits = sms / tiles;
        splits = splits < 1 ? 1 : splits > s.Chunks ? s.Chunks : splits;
        s.Per = (s.Chunks + splits - 1) / splits;
        s.Splits = (s.Chunks + s.Per - 1) / s.Per;
        return s;
    };
    p.Shape[PH_PROJ] = shape(4 * ((hs + 127) / 128), d.dim);
    p.Shape[PH_COMB] = shape(d.dim / 128, 4 * hs);
    p.Shape[PH_EXPAND] = shape(d.relu_dim / 128, d.dim);
    p.Shape[PH_CONTRACT] = shape(d.dim / 128, d.relu_dim);
    p.NSeq = nSeq;
    p.Dim = d.dim;
    p.Heads = d.head_count;
    p.HeadSize = D;
    p.PerGroup = AttGroupHeads(d.head_count, D);
    p.HeadGroups = (d.head_count + p.PerGroup - 1) / p.PerGroup;
    const int perLoad = 512 / D / p.PerGroup; // a power of two for every size of a group
    p.PerLoadLog = perLoad >= 8 ? 3 : perLoad >= 4 ? 2 : perLoad >= 2 ? 1 : 0;
    // as the decode kernel's four warps share the heads of a chunk, 512 columns each
    const int wide = (hs + 511) / 512;
    p.Split = wide == 1 ? 4 : wide == 2 ? 2 : 1;
    p.ReluDim = d.relu_dim;
    p.Capacity = capacity;
    p.MaxCtx = maxCtx + 1;
    p.RopeLen = model->rope_len;
    p.Labels = labels;
    p.LabelsPerSeq = labelsPerSeq;
    p.LabelCount = d.label_count;
    p.Embed = model->label_embed;
    p.EmbedScale = model->label_embed_scale;
    p.Rope = model->rope;
    p.DotScale = HostAttDotScale(D);
    p.Barrier = b.Sync;
    p.Arrived = b.Sync + 64;
    p.Proj = b.Proj;
    p.Comb = b.Comb;
    p.Expand = b.Expand;
    p.Contract = b.Contract;
    p.StateA = b.StateA;
    p.StateB = b.StateB;
    p.K8 = b.K8;
    p.Kv8 = b.Kv8;
    p.NormState = b.NormState;
    p.Partial = b.Partial;
    p.Status = statusWord;
    int done = 0;
    do {
        p.LayerCount = d.layer_count - done < PS_LAYERS ? d.layer_count - done : PS_LAYERS;
        p.FirstSource = done == 0 ? SRC_EMBED : SRC_STATE;
        for (int i = 0; i < p.LayerCount; ++i) {
            const tsa_infer_layer &layer = model->layers[done + i];
            TStepLayer &t = p.Layers[i];
            const int8_t *w[7] = {layer.qk, layer.qv, layer.k, layer.v, layer.combiner, layer.expand, layer.contract};
            for (int k = 0; k < 7; ++k) {
                t.W[k] = w[k];
            }
            t.Seqs = layerSeqs[done + i];
            t.CtxLens = ctxLens + (size_t)(done + i) * nSeq;
            // same association as cpu_infer.cpp:504: qvScale *= (QVScale * VEC_SCALE) * dotScale(dim)
            t.QvMult = layer.qv_scale * INF_VEC_SCALE * sqrtf(1.0f / d.dim);
            t.CombScale = layer.combiner_scale * INF_VEC_SCALE * sqrtf(1.0f / (hs * 4));
            t.ContractScale = layer.contract_scale * INF_VEC_SCALE * sqrtf(1.0f / d.relu_dim);
            t.Slope = layer.alibi_slope;
            t.Window = layer.attention_width;
        }
        rc = CheckCuda(cudaMemsetAsync(b.Sync, 0, b.ZeroBytes, stream), "clearing the inference sums");
        if (rc == TSA_OK) {
            void *args[] = {&p};
            rc = CheckCuda(cudaLaunchCooperativeKernel(kern, dim3(sms), dim3(PS_THREADS), args, smemBytes, stream), "inference layers launch");
        }
        done += p.LayerCount;
    } while (rc == TSA_OK && done < d.layer_count);
    return rc;
}

} // namespace tsa
