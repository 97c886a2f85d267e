// The projection that feeds the attention fused with its store op: int8 activations x int8 matrix on the tensor cores,
// then per-head RMS normalise, rope and quantise in the epilogue, straight from the accumulators.
// Replaces MulForwardInt8 / MulForwardFp8 <TStoreRowTileNormalizeRope> / <TStoreRowTileNormalize> of the reference
// (code/gpt/compute/gpt_cuda.cu:488-496; store ops code/lib/cuda/cuda_matmul.cuh:147-204, rope
// code/gpt/compute/gpt_rope.cuh:4-66): the fp32 projection never goes to memory.
//
//   y[t][n]  = (float)(int32 dot of x[t] and w[n]) * srcScale      (e4m3 operands: f32 dot on the tensor cores)
//   per head: discr = sqrt(sum y^2 / D) * vecScale;  z = y / discr;  rope (elements k and k + 32 of a 64-block);
//             dst = quantise(z) (int8 or e4m3);  scale[head][t] = discr
//
// Persistent, one CTA per SM, single or in pairs (clusters of two).
// Single: a CTA takes tiles of 128 rows of x times 256 output columns (4 heads of 64 or 2 of 128), tcgen05.mma M = 128, N = 256, with a ring
// of 64-column chunks.
// Pair: a tile has 256 rows; tcgen05.mma cta_group::2, M = 256, N = 256: each CTA copies 128 rows of x and the weights of 128 columns, the
// first one issues the products, which read the operands of both, and each has the accumulators of its own rows; both CTAs' copies
// count on the first one's barriers, a commit frees a stage in both.  Chunks of 128 columns: with 64 every stage pays its round trip
// of commit, copy and barrier across the two SMs (58 us where 128 take 43 to 51).
// Either way the accumulators are 256 tensor-memory columns per CTA, two such sets in turn.  One warp of each CTA streams its operands
// through a TMA ring that runs on across tiles, one issues the MMAs, and eight warps work on the epilogue of the tile before: a row
// belongs to two threads, each with half of the tile's heads, so a head's sum of squares, the rotation partners and the 64 output
// bytes of a block are all in one thread: no exchange between threads, sums in the scalar loop's order (bit-identical to the
// stand-alone normalise + rope + quantise of the CPU code on the same projection).  Tiles in a row are neighbours along the
// columns, so the rows of x stay in L2 and the rows of the rope table in shared memory.
// What bounds it: at large inner sizes the operand stream out of L2, 24 KB for every 64 columns in a single CTA, of which pairs copy two
// thirds; at small ones the epilogue, and a pair's epilogues wait for each other.
#include "att_sm100_common.cuh"

namespace tsa {

constexpr int PROJ_M = 128, PROJ_N = 256; // rows of a CTA, columns of a tile
constexpr int PROJ_LOAD_WARP = 0, PROJ_MMA_WARP = 1, PROJ_EPI_WARPS = 8;
constexpr int PROJ_EPI_THREADS = PROJ_EPI_WARPS * 32, PROJ_THREADS = PROJ_EPI_THREADS + 64;
constexpr int PROJ_SMEM_MAX = 227 * 1024;

// Whether pairs are taken.  Below these inner sizes tiles of single CTAs were faster at some number of rows (1 to 131072), from there on
// pairs were as fast or faster at all of them.  The longer a tile's epilogue (16-bit results are twice the bytes), the later.  Single ->
// pair, 32768 rows without rope: int8 to e4m3 30.2 -> 32.1 us (768 -> 12 x 64), 40.6 -> 39.2 (1024 -> 16 x 64), 133 -> 105 (2048 -> 16 x 128);
// int8 to bf16 35.6 -> 37.8, 44.0 -> 47.0, 61.5 -> 59.1 (1280 -> 20 x 64), 147 -> 120; e4m3 to int8 with rope 37.2 -> 39.4, 49.8 -> 51.2,
// 62.0 -> 60.8 (1152 -> 18 x 64), 167 -> 149.  With no more tiles than SMs no epilogue waits for another one, and pairs win from 1024 on
// (128 rows, 1024 -> 16 x 64: 10.5 -> 10.1 us to bf16, 11.6 -> 11.3 from e4m3).
inline bool ProjInPairs(int dim, bool srcE4M3, bool dst16, long long singleTiles, int sms)
{
    return dim >= (dst16 ? 1280 : srcE4M3 ? 1152 : 1024) || (dim >= 1024 && singleTiles <= sms);
}
// what a CTA copies of a chunk: PROJ_M rows of x, W_ROWS of w, KB columns of both
template <bool PAIR>
struct TProjShape {
    static constexpr int CTAS = PAIR ? 2 : 1;
    static constexpr int KB = PAIR ? 128 : 64;
    static constexpr int W_ROWS = PROJ_N / CTAS;
    static constexpr int STAGE_BYTES = (PROJ_M + W_ROWS) * KB;
};
constexpr int PROJ_MAX_STAGES = (PROJ_SMEM_MAX - 2048) / TProjShape<false>::STAGE_BYTES;

// (without a pair the CTA itself is the first one, and the only one)
struct TProjMisc {
    uint64_t Full[PROJ_MAX_STAGES], Empty[PROJ_MAX_STAGES]; // ring: in the first CTA: the copies of both landed / MMAs that read them retired (both CTAs)
    uint64_t AccFull[2], AccEmpty[2];                       // accumulator set complete (both CTAs) / in the first CTA: read out, an arrival per epilogue warp of both
    uint64_t Drained;                                       // a wait ran out: the products issued have retired (both CTAs)
    uint32_t TmemBase;
    int Abort;        // a bounded wait ran out somewhere in the pair (both CTAs)
    int Requested[2]; // in the first CTA: chunks whose copies either one's loader has requested
    int Issued;       // chunks whose products were issued (both CTAs)
};

// arrival, with release at cluster scope, on the barrier that lies in the first CTA of the pair where `bar` lies in this one
__device__ __forceinline__ void ArriveInFirst(uint64_t *bar)
{
    asm volatile(
        "{\n\t"
        ".reg .b32 remote;\n\t"
        "mapa.shared::cluster.u32 remote, %0, 0;\n\t"
        "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [remote];\n\t"
        "}" ::"r"(SmemAddr(bar))
        : "memory");
}
// `value` into the word that lies in the given CTA of the pair where `word` lies in this one
__device__ __forceinline__ void StoreInPair(int *word, int value, int rank)
{
    asm volatile(
        "{\n\t"
        ".reg .b32 remote;\n\t"
        "mapa.shared::cluster.u32 remote, %0, %2;\n\t"
        "st.relaxed.cluster.shared::cluster.u32 [remote], %1;\n\t"
        "}" ::"r"(SmemAddr(word)),
        "r"(value), "r"(rank)
        : "memory");
}
// counts bytes as landed that nobody copies
__device__ __forceinline__ void MbarCompleteTx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.complete_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(SmemAddr(bar)), "r"(bytes) : "memory");
}
// WaitBarA for a barrier the other CTA of the pair arrives on
__device__ __forceinline__ bool WaitBarPair(uint64_t *bar, uint32_t parity, const int *abortFlag, long long limit)
{
    const long long t0 = clock64();
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 32; ++i) {
            uint32_t ok;
            asm volatile(
                "{\n\t"
                ".reg .pred p;\n\t"
                "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.b32 %0, 1, 0, p;\n\t"
                "}"
                : "=r"(ok)
                : "r"(SmemAddr(bar)), "r"(parity)
                : "memory");
            if (ok) {
                return true;
            }
        }
        if (*(const volatile int *)abortFlag || clock64() - t0 > limit) {
            return false;
        }
    }
}
// 2-D tile load into this CTA's shared memory, counted on the barrier that lies in the first CTA of the pair where `bar` lies in this one
__device__ __forceinline__ void TmaLoadPair(void *smemDst, const void *tensorMap, int x, int y, uint64_t *bar)
{
    asm volatile(
        "{\n\t"
        ".reg .b32 first;\n\t"
        "mapa.shared::cluster.u32 first, %4, 0;\n\t"
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [first];\n\t"
        "}" ::"r"(SmemAddr(smemDst)), "l"(tensorMap), "r"(x), "r"(y), "r"(SmemAddr(bar))
        : "memory");
}
__device__ __forceinline__ void PairSync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// D (M = 256: each CTA's 128 rows in its own tensor memory) (+)= A B^T, A's rows and B's rows split between the two CTAs' shared memory
template <bool E4M3>
__device__ __forceinline__ void MmaPairSS(uint32_t dTmem, uint64_t aDesc, uint64_t bDesc, uint32_t idesc, uint32_t accumulate)
{
    if (E4M3) {
        asm volatile(
            "{\n\t"
            ".reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t"
            "}" ::"r"(dTmem), "l"(aDesc), "l"(bDesc), "r"(idesc), "r"(accumulate)
            : "memory");
    } else {
        asm volatile(
            "{\n\t"
            ".reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t"
            "}" ::"r"(dTmem), "l"(aDesc), "l"(bDesc), "r"(idesc), "r"(accumulate)
            : "memory");
    }
}
// arrive on the barrier of both CTAs when all MMAs issued so far by this thread have completed
__device__ __forceinline__ void MmaCommitPair(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(SmemAddr(bar)), "h"((uint16_t)3)
                 : "memory");
}

__device__ __forceinline__ uint32_t PackBf16(float lo, float hi)
{
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&h);
}

struct TProjArgs {
    P2D<float> Rope;  // [len][D] f32, may be absent
    P2D<uint8_t> Dst; // [rows][H * D]
    P2D<float> Scale; // [H][rows], may be absent
    float VecScale, SrcScale, RopeDir;
    int Len, Rows, HeadCount, Chunks;
    int ColTiles, Items; // tiles along the output columns, and all of them
    int Stages;          // of the ring
    // self-test of the failure path: bound of every barrier wait in clock cycles (about a second in production) and the index, in a CTA's
    // own sequence, of a chunk of x that it (of a pair the second one) requests but never copies (-1: none)
    long long WaitCycles;
    int WithholdChunk;
};

// `value` into the word of one of the pair's CTAs
template <bool PAIR>
__device__ __forceinline__ void ProjStore(int *word, int value, int toRank)
{
    if constexpr (PAIR) {
        StoreInPair(word, value, toRank);
    } else {
        *(volatile int *)word = value;
    }
}
// What happens when a wait runs out is out of line: a CTA runs most of its code once, and every instruction of it has to be fetched.  Written
// out, these two functions cost 0.3 to 0.5 us of a launch that takes 8 to 12.
template <bool PAIR>
__device__ __noinline__ void ProjFail(TProjMisc &misc, int *status, int code)
{
    for (int r = 0; r < TProjShape<PAIR>::CTAS; ++r) {
        ProjStore<PAIR>(&misc.Abort, 1, r);
    }
    if (status) {
        atomicOr(status, code);
    }
}
// All threads of the pair.  What was started and nobody has waited for must not reach a CTA that has left: the products issued, the commits
// behind them, and copies of either CTA, all counted in the first one, that no product has waited for.
template <bool PAIR>
__device__ __noinline__ void ProjDrain(TProjMisc &misc, int stages, int chunks, long long waitCycles, int rank, int refilled)
{
    using SH = TProjShape<PAIR>;
    if (rank == 0 && (threadIdx.x >> 5) == PROJ_MMA_WARP && ElectOne()) { // the lane that issued the products
        if constexpr (PAIR) {
            MmaCommitPair(&misc.Drained);
        } else {
            MmaCommit(&misc.Drained);
        }
    }
    if (threadIdx.x == PROJ_LOAD_WARP * 32) {
        const int issued = misc.Issued, freed = min(issued, max(refilled, 0)), tiles = issued / chunks;
        WaitBar(&misc.Drained, 0, waitCycles);
        for (int k = max(0, freed - stages); k < freed; ++k) {
            WaitBar(&misc.Empty[k % stages], (k / stages) & 1, waitCycles);
        }
        for (int n = max(0, tiles - 2); n < tiles; ++n) {
            WaitBar(&misc.AccFull[n & 1], (n >> 1) & 1, waitCycles);
        }
        if (rank == 0) {
            const int mine = misc.Requested[0], others = misc.Requested[SH::CTAS - 1];
            for (int k = issued; k < max(mine, others); ++k) {
                uint64_t *bar = &misc.Full[k % stages];
                if (k >= mine) {
                    MbarExpectTx(bar, SH::STAGE_BYTES); // the second CTA alone requested it
                } else if (k >= others) {
                    MbarCompleteTx(bar, SH::STAGE_BYTES); // the first CTA alone
                }
                WaitBar(bar, (k / stages) & 1, waitCycles);
            }
        }
    }
    __syncthreads();
    if constexpr (PAIR) {
        PairSync();
    }
}

// X_E4M3: both operands are e4m3 bytes (MulForwardFp8, gpt_cuda.cu:488-491), products accumulate in f32 on the tensor
// cores (kind::f8f6f4); otherwise int8 x int8 with exact int32 accumulators (kind::i8).
// DST: TSA_I8, TSA_E4M3 (quantised) or TSA_F16 / TSA_BF16 (the normalised, rotated values themselves: the reference's K16).
template <int D, int DST, bool X_E4M3, bool PAIR>
__global__ void __launch_bounds__(PROJ_THREADS, 1) ProjNormRopeKernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, TProjArgs a,
    int *status)
{
    using SH = TProjShape<PAIR>;
    constexpr int CTAS = SH::CTAS, KB = SH::KB, STAGE_BYTES = SH::STAGE_BYTES;
    // s32 accumulators, s8 x s8 -- or f32 accumulators, e4m3 x e4m3; both operands K-major
    constexpr uint32_t IDESC = X_E4M3 ? MakeInstrDesc(1, 0, 0, 0, 0, CTAS * PROJ_M, PROJ_N) : MakeInstrDesc(2, 1, 1, 0, 0, CTAS * PROJ_M, PROJ_N);
    auto accValue = [](uint32_t bits) { return X_E4M3 ? __uint_as_float(bits) : (float)(int32_t)bits; };
    constexpr int HPC = PROJ_N / D;                                          // heads per tile
    extern __shared__ uint8_t projSmemRaw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)projSmemRaw + 1023) & ~(uintptr_t)1023);
    TProjMisc &misc = *reinterpret_cast<TProjMisc *>(smem + a.Stages * STAGE_BYTES);
    float *ropeTile = reinterpret_cast<float *>(smem + a.Stages * STAGE_BYTES + 1024);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = blockIdx.x % CTAS; // in the pair
    if (tid == 0) {
        for (int s = 0; s < a.Stages; ++s) {
            MbarInit(&misc.Full[s], 1);
            MbarInit(&misc.Empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            MbarInit(&misc.AccFull[b], 1);
            MbarInit(&misc.AccEmpty[b], CTAS * PROJ_EPI_WARPS);
        }
        MbarInit(&misc.Drained, 1);
        misc.Abort = 0;
        FenceBarrierInit();
    }
    if (warp == PROJ_MMA_WARP) {
        if constexpr (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(SmemAddr(&misc.TmemBase)), "r"(2 * PROJ_N) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            TmemAlloc(&misc.TmemBase, 2 * PROJ_N);
            TmemRelinquish();
        }
    }
    TcFenceBefore();
    __syncthreads();
    if constexpr (PAIR) {
        PairSync(); // the other CTA's barriers and tensor memory are set up too
    }
    TcFenceAfter();
    const uint32_t tmem = misc.TmemBase;
    PdlTrigger(); // behind the allocation: a CTA of the next kernel may hold tensor memory of this SM from here on
    PdlWait();
    const int *abortFlag = &misc.Abort;
    auto fail = [&](int code) { ProjFail<PAIR>(misc, status, code); };
    const int pair = blockIdx.x / CTAS, pairs = gridDim.x / CTAS;
    const int itemBegin = (int)((long long)a.Items * pair / pairs), itemEnd = (int)((long long)a.Items * (pair + 1) / pairs);
    const int refilled = (itemEnd - itemBegin) * a.Chunks - a.Stages; // chunks whose stage is used again: only those are reported free
    auto rowOf = [&](int item) { return (item / a.ColTiles * CTAS + rank) * PROJ_M; };
    if (warp == PROJ_LOAD_WARP) {
        if (lane == 0) {
            PrefetchTensorMap(&tmX);
            PrefetchTensorMap(&tmW);
            int s = 0, phase = 0, requested = 0; // ring slot, its parity, chunks requested
            bool failed = false;
            for (int item = itemBegin; item < itemEnd && !failed; ++item) {
                const int rowBase = rowOf(item), colBase = item % a.ColTiles * PROJ_N + rank * SH::W_ROWS;
                for (int c = 0; c < a.Chunks; ++c) {
                    if (requested >= a.Stages && !WaitBarA(&misc.Empty[s], phase ^ 1, abortFlag, a.WaitCycles)) {
                        failed = true;
                        fail(kDevTimeoutMma);
                        break;
                    }
                    uint8_t *sA = smem + s * STAGE_BYTES, *sB = sA + PROJ_M * KB;
                    if (rank == 0) {
                        MbarExpectTx(&misc.Full[s], CTAS * STAGE_BYTES);
                    }
                    const bool withheld = rank == CTAS - 1 && requested == a.WithholdChunk; // self-test: the bytes of a withheld copy never arrive
                    if constexpr (PAIR) {
                        if (!withheld) {
                            TmaLoadPair(sA, &tmX, c * KB, rowBase, &misc.Full[s]);
                        }
                        TmaLoadPair(sB, &tmW, c * KB, colBase, &misc.Full[s]);
                    } else {
                        if (!withheld) {
                            TmaLoad2D(sA, &tmX, c * KB, rowBase, &misc.Full[s]);
                        }
                        TmaLoad2D(sB, &tmW, c * KB, colBase, &misc.Full[s]);
                    }
                    ++requested;
                    if (++s == a.Stages) {
                        s = 0;
                        phase ^= 1;
                    }
                }
            }
            ProjStore<PAIR>(&misc.Requested[rank], requested, 0);
        }
        __syncwarp();
    } else if (warp == PROJ_MMA_WARP) {
        if (rank == 0) {
            // the whole warp runs the loop and the waits, one elected lane issues (descriptors stay in uniform registers that way)
            int s = 0, phase = 0, n = 0, issued = 0;
            bool failed = false;
            auto wait = [&](uint64_t *bar, uint32_t parity, int code) {
                bool ok;
                if constexpr (PAIR) {
                    ok = WaitBarPair(bar, parity, abortFlag, a.WaitCycles);
                } else {
                    ok = WaitBarA(bar, parity, abortFlag, a.WaitCycles);
                }
                if (!__all_sync(0xffffffffu, ok)) {
                    failed = true;
                    if (lane == 0) {
                        fail(code);
                    }
                }
                return !failed;
            };
            for (int item = itemBegin; item < itemEnd && !failed; ++item, ++n) {
                const uint32_t acc = tmem + (n & 1) * PROJ_N;
                if (n >= 2 && !wait(&misc.AccEmpty[n & 1], ((n >> 1) - 1) & 1, kDevTimeoutMma)) {
                    break;
                }
                for (int c = 0; c < a.Chunks; ++c) {
                    if (!wait(&misc.Full[s], phase, kDevTimeoutTma)) {
                        break;
                    }
                    TcFenceAfter();
                    if (ElectOne()) {
                        const uint32_t sA = SmemAddr(smem + s * STAGE_BYTES), sB = sA + PROJ_M * KB;
#pragma unroll
                        for (int ks = 0; ks < KB / 32; ++ks) {
                            const uint64_t aDesc = MakeSmemDesc(sA + ks * 32, 16, 8 * KB, KB);
                            const uint64_t bDesc = MakeSmemDesc(sB + ks * 32, 16, 8 * KB, KB);
                            const uint32_t accumulate = (c > 0 || ks > 0) ? 1u : 0u;
                            if constexpr (PAIR) {
                                MmaPairSS<X_E4M3>(acc, aDesc, bDesc, IDESC, accumulate);
                            } else if constexpr (X_E4M3) {
                                MmaF8SS(acc, aDesc, bDesc, IDESC, accumulate);
                            } else {
                                MmaI8SS(acc, aDesc, bDesc, IDESC, accumulate);
                            }
                        }
                        auto commit = [&](uint64_t *bar) {
                            if constexpr (PAIR) {
                                MmaCommitPair(bar);
                            } else {
                                MmaCommit(bar);
                            }
                        };
                        if (issued < refilled) { // nobody waits for a later arrival, and it could reach a CTA that has left
                            commit(&misc.Empty[s]);
                        }
                        if (c == a.Chunks - 1) {
                            commit(&misc.AccFull[n & 1]);
                        }
                    }
                    __syncwarp();
                    ++issued;
                    if (++s == a.Stages) {
                        s = 0;
                        phase ^= 1;
                    }
                }
            }
            if (lane < CTAS) {
                ProjStore<PAIR>(&misc.Issued, issued, lane);
            }
        }
        __syncwarp();
    } else {
        constexpr int BAR_EPI = 1;
        const int quad = warp & 3, colHalf = (warp - 2) >> 2; // tensor-memory lanes of the warp; two threads per row: each takes half of the tile's heads
        const int rowInTile = quad * 32 + lane;
        const bool withRope = a.Rope.Valid();
        // 32 bytes of a row: one store (a whole sector) where the rows allow it
        const bool wideStores = (((uintptr_t)a.Dst.Data | (uintptr_t)a.Dst.Stride) & 31) == 0;
        auto store32 = [&](uint8_t *dst, const uint32_t *w) {
            if (wideStores) {
                StGlobal256(dst, w);
            } else {
                reinterpret_cast<uint4 *>(dst)[0] = make_uint4(w[0], w[1], w[2], w[3]);
                reinterpret_cast<uint4 *>(dst)[1] = make_uint4(w[4], w[5], w[6], w[7]);
            }
        };
        int ropeRow = -1, n = 0; // first row of the rope table's rows in shared memory
        bool failed = false;
        for (int item = itemBegin; item < itemEnd; ++item, ++n) {
            const int rowBase = rowOf(item), headBase = item % a.ColTiles * HPC;
            if (!WaitBarA(&misc.AccFull[n & 1], (n >> 1) & 1, abortFlag, a.WaitCycles)) {
                failed = true;
                fail(kDevTimeoutMma);
            }
            // one vote of the epilogue threads per tile, so that they leave together; it also says that all of them are done with the rope
            // rows of the tile before
            if (BarRedOr(BAR_EPI, PROJ_EPI_THREADS, failed)) {
                break;
            }
            TcFenceAfter();
            // every thread of a warp takes part in the tensor-memory loads (they are warp-wide instructions): rows past the
            // buffer only skip their global loads and stores
            const int t = rowBase + rowInTile;
            const bool inBuf = t < a.Rows;
            // the rows of the rope table through shared memory: coalesced loads, and a row pitch of D + 1 words lets every thread walk its
            // own row without bank conflicts
            if (withRope && ropeRow != rowBase) {
                ropeRow = rowBase;
#pragma unroll 4
                for (int idx = tid - 64; idx < PROJ_M * (D / 4); idx += PROJ_EPI_THREADS) {
                    const int row = idx / (D / 4), c4 = idx - row * (D / 4);
                    float4 v = make_float4(0, 0, 0, 0);
                    if (rowBase + row < a.Len) {
                        v = *reinterpret_cast<const float4 *>(a.Rope.Row(rowBase + row) + c4 * 4);
                    }
                    float *dstRope = ropeTile + row * (D + 1) + c4 * 4;
                    dstRope[0] = v.x, dstRope[1] = v.y, dstRope[2] = v.z, dstRope[3] = v.w;
                }
                BarSync(BAR_EPI, PROJ_EPI_THREADS);
            }
            {
                const uint32_t tLane = tmem + (n & 1) * PROJ_N + ((uint32_t)(quad * 32) << 16);
                const bool live = t < a.Len;
#pragma unroll 1
                for (int hh = colHalf * (HPC / 2); hh < (colHalf + 1) * (HPC / 2); ++hh) {
                    const int head = headBase + hh;
                    if (head >= a.HeadCount) {
                        break;
                    }
                    // sum of squares of the head in column order, one rounding per product and per sum
                    float sum2 = 0;
#pragma unroll 1
                    for (int c0 = 0; c0 < D; c0 += 32) {
                        uint32_t r[32];
                        TmemLd32(tLane + hh * D + c0, r);
                        TmemWaitLd();
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            const float y = __fmul_rn(accValue(r[i]), a.SrcScale);
                            sum2 = __fadd_rn(sum2, __fmul_rn(y, y));
                        }
                    }
                    float discr = 0;
                    if (sum2 > 0 && live) {
                        discr = __fmul_rn(__fsqrt_rn(__fdiv_rn(sum2, (float)D)), a.VecScale);
                    }
                    const float mult = discr > 0 ? __fdiv_rn(1.0f, discr) : 0.0f;
                    constexpr int ES = (DST == TSA_F16 || DST == TSA_BF16) ? 2 : 1; // bytes per output element
                    uint8_t *dstRow = a.Dst.Row(inBuf ? t : 0) + head * D * ES;
#pragma unroll 1
                    for (int blk = 0; blk < D; blk += 64) {
                        uint32_t lo[32], hi[32];
                        TmemLd32(tLane + hh * D + blk, lo);
                        TmemLd32(tLane + hh * D + blk + 32, hi);
                        TmemWaitLd();
                        uint32_t outLo[8], outHi[8];
#pragma unroll
                        for (int q = 0; q < 8; ++q) {
                            float z0[4], z1[4];
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const int k = q * 4 + i;
                                float y0 = __fmul_rn(__fmul_rn(accValue(lo[k]), a.SrcScale), mult);
                                float y1 = __fmul_rn(__fmul_rn(accValue(hi[k]), a.SrcScale), mult);
                                if (withRope && live) {
                                    const float cs = ropeTile[rowInTile * (D + 1) + blk + k];
                                    const float sn = __fmul_rn(ropeTile[rowInTile * (D + 1) + blk + k + 32], a.RopeDir);
                                    const float r0 = __fsub_rn(__fmul_rn(y0, cs), __fmul_rn(y1, sn));
                                    const float r1 = __fadd_rn(__fmul_rn(y0, sn), __fmul_rn(y1, cs));
                                    y0 = r0;
                                    y1 = r1;
                                }
                                z0[i] = y0;
                                z1[i] = y1;
                            }
                            if (ES == 2) {
                                // eight words = 16 columns = 32 bytes at a time
                                const int w0 = 2 * (q & 3);
                                if (DST == TSA_F16) {
                                    outLo[w0] = PackHalf2(z0[0], z0[1]), outLo[w0 + 1] = PackHalf2(z0[2], z0[3]);
                                    outHi[w0] = PackHalf2(z1[0], z1[1]), outHi[w0 + 1] = PackHalf2(z1[2], z1[3]);
                                } else {
                                    outLo[w0] = PackBf16(z0[0], z0[1]), outLo[w0 + 1] = PackBf16(z0[2], z0[3]);
                                    outHi[w0] = PackBf16(z1[0], z1[1]), outHi[w0 + 1] = PackBf16(z1[2], z1[3]);
                                }
                                if ((q & 3) == 3 && inBuf) {
                                    store32(dstRow + (blk + (q - 3) * 4) * 2, outLo);
                                    store32(dstRow + (blk + 32 + (q - 3) * 4) * 2, outHi);
                                }
                            } else if (DST == TSA_E4M3) {
                                outLo[q] = PackE4M3x4(z0[0], z0[1], z0[2], z0[3]);
                                outHi[q] = PackE4M3x4(z1[0], z1[1], z1[2], z1[3]);
                            } else {
                                outLo[q] = 0;
                                outHi[q] = 0;
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
                                    outLo[q] |= (uint32_t)(FloatToI8Sat(z0[i]) & 0xff) << (8 * i);
                                    outHi[q] |= (uint32_t)(FloatToI8Sat(z1[i]) & 0xff) << (8 * i);
                                }
                            }
                        }
                        if (inBuf && ES == 1) {
                            store32(dstRow + blk, outLo);
                            store32(dstRow + blk + 32, outHi);
                        }
                    }
                    if (a.Scale.Valid() && inBuf) {
                        a.Scale.Row(head)[t] = discr;
                    }
                }
            }
            // this warp has read the accumulators for the last time
            TcFenceBefore();
            __syncwarp();
            if (lane == 0) {
                if constexpr (PAIR) {
                    ArriveInFirst(&misc.AccEmpty[n & 1]);
                } else {
                    MbarArrive(&misc.AccEmpty[n & 1]);
                }
            }
        }
    }
    TcFenceBefore();
    __syncthreads();
    if constexpr (PAIR) {
        PairSync(); // neither CTA leaves while the other may still arrive on its barriers
    }
    if (*(volatile int *)&misc.Abort) { // which both CTAs see alike here
        ProjDrain<PAIR>(misc, a.Stages, a.Chunks, a.WaitCycles, rank, refilled);
    }
    if (warp == PROJ_MMA_WARP) {
        if constexpr (PAIR) {
            asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * PROJ_N) : "memory");
        } else {
            TmemDealloc(tmem, 2 * PROJ_N);
        }
    }
}

} // namespace tsa

using namespace tsa;

extern "C" __attribute__((visibility("default"))) int tsa_matmul_norm_rope_quant(int srcDtype, int dstDtype, float vecScale, float srcScale, tsa_ptr2d x, tsa_ptr2d w,
    tsa_ptr2d rope, float ropeDir, tsa_ptr2d dst, tsa_ptr2d scale, int headCount, int headDim, int len, int *statusWord, tsa_stream_t stream)
{
    TSA_REQUIRE(srcDtype == TSA_I8 || srcDtype == TSA_E4M3, "tsa_matmul_norm_rope_quant: x and w must both be i8 or both e4m3");
    TSA_REQUIRE(dstDtype == TSA_I8 || dstDtype == TSA_E4M3 || dstDtype == TSA_F16 || dstDtype == TSA_BF16,
        "tsa_matmul_norm_rope_quant: dst dtype must be i8, e4m3, f16 or bf16");
    TSA_REQUIRE(x.data && w.data && dst.data, "tsa_matmul_norm_rope_quant: null x / w / dst");
    TSA_REQUIRE(headCount > 0 && (headDim == 64 || headDim == 128), "tsa_matmul_norm_rope_quant: head size %d must be 64 or 128", headDim);
    const int dim = x.xsize, outCols = headCount * headDim;
    TSA_REQUIRE(dim > 0 && dim % 64 == 0 && w.xsize == dim, "tsa_matmul_norm_rope_quant: inner size %d (x) / %d (w) must be equal multiples of 64", dim,
        w.xsize);
    TSA_REQUIRE(w.ysize >= outCols && dst.xsize >= outCols, "tsa_matmul_norm_rope_quant: w has %d rows, dst %d columns, H*D = %d", w.ysize, dst.xsize, outCols);
    TSA_REQUIRE(len >= 0 && len <= x.ysize && len <= dst.ysize, "tsa_matmul_norm_rope_quant: len %d exceeds buffers (%d, %d rows)", len, x.ysize, dst.ysize);
    TSA_REQUIRE((uintptr_t)x.data % 16 == 0 && x.stride_bytes % 16 == 0 && (uintptr_t)w.data % 16 == 0 && w.stride_bytes % 16 == 0 &&
            (uintptr_t)dst.data % 16 == 0 && dst.stride_bytes % 16 == 0,
        "tsa_matmul_norm_rope_quant: x, w and dst must be 16-byte aligned with 16-byte multiples as row strides");
    if (scale.data) {
        TSA_REQUIRE(scale.ysize >= headCount && scale.xsize >= dst.ysize, "tsa_matmul_norm_rope_quant: scale plane too small");
    }
    if (rope.data) {
        TSA_REQUIRE(rope.xsize >= headDim && rope.ysize >= len, "tsa_matmul_norm_rope_quant: rope table smaller than [len][headDim]");
        TSA_REQUIRE((uintptr_t)rope.data % 16 == 0 && rope.stride_bytes % 16 == 0, "tsa_matmul_norm_rope_quant: rope table must be 16-byte aligned");
    }
    if (dst.ysize == 0) {
        return TSA_OK;
    }
    int dev = 0, sms = 0;
    int rc = CheckCuda(cudaGetDevice(&dev), "cudaGetDevice");
    if (rc == TSA_OK) {
        rc = CheckCuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "cudaDeviceGetAttribute");
    }
    if (rc != TSA_OK) {
        return rc;
    }
    const int colTiles = (outCols + PROJ_N - 1) / PROJ_N;
    const bool pair = ProjInPairs(dim, srcDtype == TSA_E4M3, dstDtype == TSA_F16 || dstDtype == TSA_BF16, (long long)((dst.ysize + PROJ_M - 1) / PROJ_M) * colTiles, sms);
    const int ctas = pair ? 2 : 1, kb = pair ? TProjShape<true>::KB : TProjShape<false>::KB;
    const int stageBytes = pair ? TProjShape<true>::STAGE_BYTES : TProjShape<false>::STAGE_BYTES;
    CUtensorMap mx, mw;
    tsa_ptr2d xv = x;
    xv.ysize = len; // rows past len read as zeros
    rc = len > 0 ? MakeTileMapEx(&mx, xv, 1, kb, PROJ_M, "x") : MakeTileMapEx(&mx, x, 1, kb, PROJ_M, "x");
    if (rc == TSA_OK) {
        tsa_ptr2d wv = w;
        wv.ysize = outCols;
        rc = MakeTileMapEx(&mw, wv, 1, kb, PROJ_N / ctas, "w");
    }
    if (rc != TSA_OK) {
        return rc;
    }
    TProjArgs a;
    a.Rope = P2D<float>(rope);
    a.Dst = P2D<uint8_t>(dst);
    a.Scale = P2D<float>(scale);
    a.VecScale = vecScale;
    a.SrcScale = srcScale;
    a.RopeDir = ropeDir;
    a.Len = len;
    a.Rows = dst.ysize;
    a.HeadCount = headCount;
    a.Chunks = (dim + kb - 1) / kb; // columns past the end read as zeros
    a.ColTiles = colTiles;
    a.Items = (dst.ysize + ctas * PROJ_M - 1) / (ctas * PROJ_M) * colTiles;
    // as many ring stages as fit beside the rope rows
    const int ropeBytes = rope.data ? PROJ_M * (headDim + 1) * (int)sizeof(float) : 0;
    a.Stages = (PROJ_SMEM_MAX - 2048 - ropeBytes) / stageBytes; // at most PROJ_MAX_STAGES
    a.WaitCycles = TestHooks().WaitCycles > 0 ? TestHooks().WaitCycles : WAIT_CYCLES;
    a.WithholdChunk = TestHooks().WithholdTile;
    const int smemBytes = a.Stages * stageBytes + 1024 /* barriers */ + 1024 /* alignment */ + ropeBytes;
    const bool x8 = srcDtype == TSA_E4M3;
    const void *kern = nullptr;
#define TSA_PROJ_CASE(DD, DT, X8)                                                                                             \
    if (headDim == DD && dstDtype == DT && x8 == X8) {                                                                        \
        kern = pair ? (const void *)ProjNormRopeKernel<DD, DT, X8, true> : (const void *)ProjNormRopeKernel<DD, DT, X8, false>; \
    }
#define TSA_PROJ_CASES(DD, X8) TSA_PROJ_CASE(DD, TSA_I8, X8) TSA_PROJ_CASE(DD, TSA_E4M3, X8) TSA_PROJ_CASE(DD, TSA_F16, X8) TSA_PROJ_CASE(DD, TSA_BF16, X8)
    TSA_PROJ_CASES(64, false)
    TSA_PROJ_CASES(64, true)
    TSA_PROJ_CASES(128, false)
    TSA_PROJ_CASES(128, true)
#undef TSA_PROJ_CASES
#undef TSA_PROJ_CASE
    rc = CheckCuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smemBytes), "cudaFuncSetAttribute");
    if (rc != TSA_OK) {
        return rc;
    }
    void *args[] = {&mx, &mw, &a, &statusWord};
    return CheckCuda(LaunchPdl(kern, dim3(ctas * (a.Items < sms / ctas ? a.Items : sms / ctas)), dim3(PROJ_THREADS), smemBytes, (cudaStream_t)stream, args, ctas), "tsa_matmul_norm_rope_quant launch");
}
