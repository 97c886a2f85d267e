// Quantized attention backward for sm_100a on the tensor cores (tcgen05, bf16 operands, f32 accumulators in
// tensor memory).
//
// Replaces Fp8AttGradQK / Fp8AttGradQV (code/gpt/compute/gpt_att_fp8.cuh:277-983) and Fp16AttGradQK / QV
// (gpt_att_fp16.cuh:332-616).  Math (TAttentionComputer::CalcDDot / GradQK / GradQV, gpt_cpu.cpp:465-555):
//   z_ij = dot(q8_i, k8_j) sq_i sk_j c - slope (i - j);   p_ij = 2^(z_ij - lse_i)
//   dP_ij = dO_i . (sv_j v8_j);   dS_ij = p_ij (dP_ij - delta_i) c ln2
//   dq_i = sum_j dS_ij sk_j k8_j;   dk_j = sum_i dS_ij sq_i q8_i;   dv_j = sum_i p_ij dO_i
// The reference quantises dS to e4m3 with a two-pass row maximum (doc/precision.md:44); here the stored 8-bit
// vectors are first widened to bf16 (exact: every int8 and e4m3 value is a bf16 number) into scratch, dO is taken
// as bf16, and all GEMMs run as kind::f16 with dS and P handed to the tensor core as bf16: one pass, no row maximum.
//
// One kernel, two modes, the same tile engine; a work item is a head and 128 rows:
//   mode dQ     : item = head x 128 query rows (R1 = Q, R2 = dO), loop over key tiles (C1 = K, C2 = V) of the row
//                 spans:  S = R1 C1^T, dP = R2 C2^T, A1 = dS * sk_j,                  dQ  += A1 C1
//   mode dK,dV  : item = head x 128 key rows (R1 = K, R2 = V ), loop over query tiles (C1 = Q, C2 = dO) of the
//                 transposed spans:  S^T = R1 C1^T, dP^T = R2 C2^T, A1 = dS * sq_i, A2 = P,  dK += A1 C1, dV += A2 C2
// Tensor memory (512 columns): [0,128) S, [128,256) dP, [256,256+D) first output, [256+D,256+2D) second output.
// A1 / A2 (bf16, two per column) are written back over the S / dP columns the writing thread has already consumed.
//
// A tile is worked on as two 64-column halves with their own barriers, so the tensor pipe and the arithmetic
// overlap: while the 16 arithmetic warps turn S / dP of one half into A1 / A2 (four threads per tile row, 16 columns
// each; packed f32x2 arithmetic on per-column factors staged in shared memory one tile ahead), the MMAs of the other
// half (its output products, then its S / dP of the next tile) run.  Each half has its own MMA-issuing warp (an elected
// lane of a converged warp issues, in grouped asm blocks); the two take turns block by block, so one does its waits
// while the other issues and the accumulation order is fixed; one more warp issues the TMA copies.  Row tiles stay in shared memory; column tiles stream through a ring of
// half stages (64 rows of C1 and C2), freed per half.
//
// Persistent: one CTA per SM (all of its tensor memory and most of its shared memory) takes items from a counter, long ones first,
// and the pipelines run on across items: the next item's row tiles are loaded when the present one's last score products have retired,
// its first scores run while the arithmetic warps still drain the outputs, and those warps look up the next item's spans while the
// last output products run.  With a CTA per item every item paid 4.4 K clocks of start-up and 7 K from its last weights to the end
// of the CTA, half of the 22 K that an item of a window-256 layer took.  All waits are bounded; a failed wait is carried to the
// arithmetic threads' next named barrier so they leave together.
#include "att_sm100_common.cuh"

namespace tsa {

constexpr int BWD_ARITH_THREADS = 512;
constexpr int BWD_CTRL_WARP = BWD_ARITH_THREADS / 32; // and the next one: control warp h issues the products of half h
constexpr int BWD_LOAD_WARP = BWD_CTRL_WARP + 2;
constexpr int BWD_THREADS = BWD_ARITH_THREADS + 96;
constexpr uint32_t BWD_TMEM_COLS = 512;
constexpr uint32_t BWD_S_COL = 0, BWD_DP_COL = 128, BWD_OUT_COL = 256;

struct TBwdParams {
    int HeadCount;
    int Rows;         // rows of every matrix
    int LenAttTiles;  // number of 64-row span blocks
    const tsa_span_group *Spans; // spans of the rows of this mode (forward spans for dQ, transposed for dK/dV)
    const int *SpanPtr;
    P2D<float> QScale, KScale, VScale;
    float QkVecScale, VVecScale;
    P2D<float> Lse, DScale;
    const float *GlobalScale;
    float C;
    float Slope;
    float GradMult;
    P2D<char> Out1, Out2;
    int WideStores;   // the outputs' rows are 32-byte aligned
    int GradDtype;
    int Items;        // row tiles x heads
    int Ascending;    // order of the row tiles: the long ones come first
    int *Counter;     // work-item counter, zero at launch
    int *Status;
    // self-test of the failure path: bound, in clock cycles, of the wait for a tile's column factors (about a second in production) and
    // which of a CTA's first two tiles has its factors staged but never announced (-1: neither): its barrier expects one arrival more (a look
    // at the tile's index in front of the arrival took 0.6 % of the kernel's time)
    long long WaitCycles;
    int WithholdTile;
};

template <int D>
struct TBwdSmem {
    static constexpr int STAGES = (D == 64) ? 3 : 2;
    static constexpr int TILE_BYTES = 128 * D * 2;
    // column tiles travel in halves of 64 rows: a ring of HSTAGES half stages, each [C1 half][C2 half]
    static constexpr int HSTAGES = 2 * STAGES;
    static constexpr int HALF_TILE_BYTES = TILE_BYTES / 2;
    static constexpr int R1_OFF = 0;
    static constexpr int R2_OFF = TILE_BYTES;
    static constexpr int C_OFF = 2 * TILE_BYTES;              // half stage s: C1 rows at C_OFF + s * TILE, C2 rows right after
    static constexpr int MISC_OFF = C_OFF + STAGES * 2 * TILE_BYTES;
    static constexpr int TOTAL = MISC_OFF + 8192;
};

struct TBwdMisc {
    // per column of the tile, double buffered by tile parity, written by the half that uses them:
    float ColA[2][TILE_ROWS]; // scale of the column vector (dQ: sk_j, dK/dV: sq_i)
    float ColT[2][TILE_ROWS]; // additive term of the exponent (dQ: ALiBi column part, dK/dV: -lse_i - ALiBi column part)
    float ColB[2][TILE_ROWS]; // dQ: sv_j c ln2;  dK/dV: -delta_i c ln2
    int Abort;
    int Turn;                 // issue blocks handed to the tensor pipe so far: control warp h issues the blocks with index = h (mod 2)
    uint64_t ItemFull[2];     // loader -> all: Item[] holds the next work item
    uint64_t ItemEmpty[2];    // all -> loader: the record has been read
    struct {
        int RowTile, Head; // RowTile < 0: no items left
        TTileIter First;   // at the item's first column tile
    } Item[2];
    uint64_t BarR;            // TMA: row tiles landed
    uint64_t BarREmpty;       // MMA warps -> loader: the item's last score products have retired
    uint64_t BarFull[8];      // TMA: half stage (64 rows of C1 and C2) landed
    uint64_t BarEmpty[8];     // MMA warp -> loader: the half stage's output products have retired
    uint64_t BarS[2];         // control -> half h: S and dP columns of the half ready
    uint64_t BarP[2];         // half h -> control: A1 / A2 of the half written (an arrival per arithmetic warp)
    uint64_t ColFull[2];      // first four arithmetic warps -> all of them: the column factors of a tile are staged
    uint64_t BarOut;          // MMA warps -> arithmetic: every output product of the item has retired
    uint32_t TmemBase;
};
static_assert(sizeof(TBwdMisc) <= 8192, "misc block");

__device__ __forceinline__ uint32_t PackBf16x2(float lo, float hi)
{
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t *>(&h);
}

// MODE_DKV = false: dQ pass; true: dK/dV pass
template <int D, bool MODE_DKV>
__global__ void __launch_bounds__(BWD_THREADS, 1) BwdSm100Kernel(const __grid_constant__ CUtensorMap tmR1,
    const __grid_constant__ CUtensorMap tmR2, const __grid_constant__ CUtensorMap tmC1, const __grid_constant__ CUtensorMap tmC2,
    const __grid_constant__ TBwdParams p)
{
    using SM = TBwdSmem<D>;
    constexpr int HSTAGES = SM::HSTAGES;
    constexpr uint32_t HALF_BLOCK_BYTES = 64 * 128;     // one [64 rows][128 bytes] block of a half column tile
    constexpr int KBLOCKS = D / 64;                     // 64-element (128-byte) blocks along the head dimension
    constexpr uint32_t BLOCK_BYTES = 128 * 128;         // one [128 rows][128 bytes] block of a tile
    constexpr uint32_t IDESC_SS = MakeInstrDesc(1, 1, 1, 0, 0, TILE_ROWS, 64); // bf16 x bf16 -> f32, both K-major, 64 columns
    constexpr uint32_t IDESC_OUT = MakeInstrDesc(1, 1, 1, 0, 1, TILE_ROWS, D); // A from tensor memory, B MN-major
    constexpr int BAR_ARITH = 1;                        // named barrier of the 512 arithmetic threads
    constexpr int QUARTER_D = D / 4;
    constexpr int OUTPUTS = MODE_DKV ? 2 : 1;

    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t *sR1 = smem + SM::R1_OFF;
    uint8_t *sR2 = smem + SM::R2_OFF;
    uint8_t *sC = smem + SM::C_OFF;
    TBwdMisc &misc = *reinterpret_cast<TBwdMisc *>(smem + SM::MISC_OFF);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // item -> row tile and head: heads side by side, long row tiles first (the late ones of the mask, the early ones of its transpose)
    auto locate = [&](int item, int &rowTile, int &head) {
        const int k = item / p.HeadCount;
        head = item - k * p.HeadCount;
        rowTile = p.Ascending ? k : p.Items / p.HeadCount - 1 - k;
    };

    if ((SmemAddr(smem) & 1023u) != 0) {
        if (tid == 0 && p.Status) {
            atomicOr(p.Status, kDevBadSpan);
        }
        return;
    }
    if (tid == 0) {
        for (int s = 0; s < 2; ++s) {
            MbarInit(&misc.ItemFull[s], 1);
            MbarInit(&misc.ItemEmpty[s], BWD_ARITH_THREADS / 32 + 2);
        }
        MbarInit(&misc.BarR, 1);
        MbarInit(&misc.BarREmpty, 2);
        for (int s = 0; s < HSTAGES; ++s) {
            MbarInit(&misc.BarFull[s], 1);
            MbarInit(&misc.BarEmpty[s], 1);
        }
        for (int h = 0; h < 2; ++h) {
            MbarInit(&misc.BarS[h], 1);
            MbarInit(&misc.BarP[h], BWD_ARITH_THREADS / 32);
        }
        for (int b = 0; b < 2; ++b) {
            MbarInit(&misc.ColFull[b], TILE_ROWS / 32 + (b == p.WithholdTile ? 1 : 0));
        }
        MbarInit(&misc.BarOut, 2);
        misc.Abort = 0;
        misc.Turn = 0;
        FenceBarrierInit();
    }
    if (warp == BWD_CTRL_WARP) {
        TmemAlloc(&misc.TmemBase, BWD_TMEM_COLS);
        TmemRelinquish();
    }
    TcFenceBefore();
    __syncthreads();
    TcFenceAfter();
    const uint32_t tmem = misc.TmemBase;
    const int *abortFlag = &misc.Abort;
    // The dK/dV pass reads nothing that the dQ pass in front of it writes: its CTAs move in as the dQ pass's leave.  They start only
    // when every dQ CTA has passed the wait here, so what the kernels before that wrote is complete and visible; the wait at the end
    // keeps the order for whatever comes behind.
    if (!MODE_DKV) {
        PdlWait();
    }
    PdlTrigger();

    if (warp == BWD_LOAD_WARP) {
        // ---------------------------------------------------------------- loader warp: the work items and every TMA copy
        if (lane == 0) {
            PrefetchTensorMap(&tmR1);
            PrefetchTensorMap(&tmR2);
            PrefetchTensorMap(&tmC1);
            PrefetchTensorMap(&tmC2);
            int g = 0, rCount = 0; // half stages / row tiles requested
            bool failed = false;
            auto wait = [&](uint64_t *bar, uint32_t parity) {
                if (!WaitBarA(bar, parity, abortFlag)) {
                    failed = true;
                    *(volatile int *)&misc.Abort = 1;
                    if (p.Status) {
                        atomicOr(p.Status, kDevTimeoutMma);
                    }
                }
                return !failed;
            };
            int item = blockIdx.x;
            for (int n = 0;; ++n) {
                if (n >= 2 && !wait(&misc.ItemEmpty[n & 1], ((n >> 1) - 1) & 1)) {
                    break;
                }
                if (item >= p.Items) {
                    misc.Item[n & 1].RowTile = -1;
                    MbarArrive(&misc.ItemFull[n & 1]);
                    break;
                }
                const int next = gridDim.x + atomicAdd(p.Counter, 1); // in flight while this item is set up
                int rowTile, head;
                locate(item, rowTile, head);
                item = next;
                TTileIter prod;
                prod.Init(p.Spans, p.SpanPtr, p.LenAttTiles, rowTile, p.Rows);
                misc.Item[n & 1].RowTile = rowTile;
                misc.Item[n & 1].Head = head;
                misc.Item[n & 1].First = prod;
                MbarArrive(&misc.ItemFull[n & 1]);
                if (!prod.Valid) {
                    continue;
                }
                // the row tiles' buffers are in use for a while yet: bring the tiles as far as L2 meanwhile
#pragma unroll
                for (int kb = 0; kb < KBLOCKS; ++kb) {
                    TmaPrefetch2D(&tmR1, head * D + kb * 64, rowTile * TILE_ROWS);
                    TmaPrefetch2D(&tmR1, head * D + kb * 64, rowTile * TILE_ROWS + 64);
                    TmaPrefetch2D(&tmR2, head * D + kb * 64, rowTile * TILE_ROWS);
                    TmaPrefetch2D(&tmR2, head * D + kb * 64, rowTile * TILE_ROWS + 64);
                }
                if (rCount > 0 && !wait(&misc.BarREmpty, (rCount - 1) & 1)) {
                    break;
                }
                // every tensor map has boxes of 64 rows x 64 elements (128 bytes): a row tile is two boxes per block
                auto loadTile = [&](uint8_t *dst, const CUtensorMap *tm) {
#pragma unroll
                    for (int kb = 0; kb < KBLOCKS; ++kb) {
                        TmaLoad2D(dst + kb * BLOCK_BYTES, tm, head * D + kb * 64, rowTile * TILE_ROWS, &misc.BarR);
                        TmaLoad2D(dst + kb * BLOCK_BYTES + HALF_BLOCK_BYTES, tm, head * D + kb * 64, rowTile * TILE_ROWS + 64, &misc.BarR);
                    }
                };
                MbarExpectTx(&misc.BarR, 2 * SM::TILE_BYTES);
                loadTile(sR1, &tmR1);
                loadTile(sR2, &tmR2);
                ++rCount;
                auto loadHalf = [&](uint8_t *dst, const CUtensorMap *tm, int rowBase, uint64_t *bar) {
#pragma unroll
                    for (int kb = 0; kb < KBLOCKS; ++kb) {
                        TmaLoad2D(dst + kb * HALF_BLOCK_BYTES, tm, head * D + kb * 64, rowBase, bar);
                    }
                };
                for (; prod.Valid && !failed; prod.Advance()) {
#pragma unroll 1
                    for (int h = 0; h < 2; ++h, ++g) {
                        const int slot = g % HSTAGES;
                        if (g >= HSTAGES && !wait(&misc.BarEmpty[slot], ((g / HSTAGES) - 1) & 1)) {
                            break;
                        }
                        MbarExpectTx(&misc.BarFull[slot], 2 * SM::HALF_TILE_BYTES);
                        loadHalf(sC + slot * 2 * SM::HALF_TILE_BYTES, &tmC1, prod.J0 + 64 * h, &misc.BarFull[slot]);
                        loadHalf(sC + slot * 2 * SM::HALF_TILE_BYTES + SM::HALF_TILE_BYTES, &tmC2, prod.J0 + 64 * h, &misc.BarFull[slot]);
                    }
                }
                if (failed) {
                    break;
                }
            }
            if (failed || *(volatile int *)&misc.Abort) {
                // drain copies that were requested, so none lands after the CTA is gone
                if (rCount > 0) {
                    WaitBar(&misc.BarR, (rCount - 1) & 1);
                }
                for (int t = max(0, g - HSTAGES); t < g; ++t) {
                    WaitBar(&misc.BarFull[t % HSTAGES], (t / HSTAGES) & 1);
                }
            }
        }
        __syncwarp();
    } else if (warp == BWD_CTRL_WARP || warp == BWD_CTRL_WARP + 1) {
        // ---------------------------------------------------------------- two MMA warps, one per 64-column half of the
        // tiles: the whole warp runs the loop and the waits, one elected lane issues (descriptors stay in uniform
        // registers that way).  The halves share nothing but the output accumulators, which the arithmetic threads
        // clear before their first hand-over so that every output product accumulates, whichever warp comes first; while
        // one warp is between two issue blocks (waits, votes, loop code) the other keeps the tensor pipe fed.
        const int h = warp - BWD_CTRL_WARP;
        {
            const uint32_t sR1a = SmemAddr(sR1), sR2a = SmemAddr(sR2), sCa = SmemAddr(sC);
            bool failed = false;
            // descriptors of a K-major tile and of an MN-major half column tile without the address (added per use, in
            // 16-byte units)
            const uint64_t kDescBase = MakeSmemDesc(0, 16, 1024, 128), mnDescBase = MakeSmemDesc(0, HALF_BLOCK_BYTES, 1024, 128);
            // columns [64h, 64h + 64) of S = R1 C1^T and dP = R2 C2^T from half stage `slot` (the 64 rows of C1 and C2 that
            // belong to the half): both operands K-major, D / 16 steps of 16 elements (32 bytes), the B blocks 8 KB apart
            auto issueScores = [&](int slot, int h) {
                const uint32_t c1 = sCa + slot * 2 * SM::HALF_TILE_BYTES, c2 = c1 + SM::HALF_TILE_BYTES;
                MmaGroupF16SS<D / 16>(tmem + BWD_S_COL + h * 64, kDescBase + (sR1a >> 4), kDescBase + (c1 >> 4), IDESC_SS, HALF_BLOCK_BYTES >> 4);
                MmaGroupF16SS<D / 16>(tmem + BWD_DP_COL + h * 64, kDescBase + (sR2a >> 4), kDescBase + (c2 >> 4), IDESC_SS, HALF_BLOCK_BYTES >> 4);
            };
            // out1 += A1 C1 (and out2 += A2 C2) over the half's 64 tile columns = 4 steps of 16: A from tensor memory
            // (the bf16 pairs of tile columns [16k, 16k + 16) sit in columns 16k .. 16k+7), B = the half column tile read
            // MN-major (16 rows of 128 bytes per step)
            auto issueOutputs = [&](int slot, int h) {
                const uint32_t c1 = sCa + slot * 2 * SM::HALF_TILE_BYTES, c2 = c1 + SM::HALF_TILE_BYTES;
                MmaQuadF16TS(tmem + BWD_OUT_COL, tmem + BWD_S_COL + h * 64, mnDescBase + (c1 >> 4), IDESC_OUT, 1u);
                if (MODE_DKV) {
                    MmaQuadF16TS(tmem + BWD_OUT_COL + D, tmem + BWD_DP_COL + h * 64, mnDescBase + (c2 >> 4), IDESC_OUT, 1u);
                }
            };
            auto fail = [&](int code) {
                failed = true;
                if (lane == 0) {
                    *(volatile int *)&misc.Abort = 1;
                    if (p.Status) {
                        atomicOr(p.Status, code);
                    }
                }
            };
            // Order inside a half: out(h, it-1) then scores(h, it): the outputs read the half's A columns before the next
            // scores overwrite them, and a thread's products run in order.  The warp never waits for its own MMAs; the
            // loader refills a half stage when the commit made after its output products completes.  Half (it, h) lives
            // in half stage (2 it + h) % HSTAGES.
            // The two warps take turns: issue blocks go to the pipe whole and in a fixed order, h0 h1 h0 h1 ..., so the
            // output accumulators, which both halves add to, receive their terms in the same order on every run (f32
            // addition does not commute with rounding: without the turns the results differed in the last bit from run
            // to run).  The waits of one warp still overlap the issue block of the other.
            auto takeTurn = [&](int index) {
                const volatile int *turn = &misc.Turn;
                if (*turn == index) {
                    return true;
                }
                const long long t0 = clock64();
                for (;;) {
#pragma unroll 1
                    for (int i = 0; i < 64; ++i) {
                        __nanosleep(20);
                        if (*turn == index) {
                            return true;
                        }
                    }
                    if (*(const volatile int *)abortFlag || clock64() - t0 > WAIT_CYCLES) {
                        return false;
                    }
                }
            };
            auto passTurn = [&](int index) {
                __syncwarp();
                if (lane == 0) {
                    *(volatile int *)&misc.Turn = index + 1;
                }
            };
            // An item's last output products are an issue block of their own, so that they do not wait for the next item's row tiles.
            int it = 0, items = 0, block = 0; // tiles, items with tiles and issue blocks so far
            for (int n = 0; !failed; ++n) {
                if (!__all_sync(0xffffffffu, WaitBarA(&misc.ItemFull[n & 1], (n >> 1) & 1, abortFlag))) {
                    fail(kDevTimeoutTma);
                    break;
                }
                const bool none = misc.Item[n & 1].RowTile < 0;
                TTileIter ctl = misc.Item[n & 1].First;
                __syncwarp();
                if (lane == 0) {
                    MbarArrive(&misc.ItemEmpty[n & 1]);
                }
                if (none) {
                    break;
                }
                if (!ctl.Valid) {
                    continue;
                }
                if (!__all_sync(0xffffffffu, WaitBarA(&misc.BarR, items & 1, abortFlag))) {
                    fail(kDevTimeoutTma);
                    break;
                }
                ++items;
                for (bool first = true;; first = false) {
                    const bool more = ctl.Valid; // a tile's scores behind the previous tile's outputs, or the item's last outputs
                    const int g = 2 * it + h;
                    const int slot = g % HSTAGES, prevSlot = (g - 2 + HSTAGES) % HSTAGES;
                    if (more) {
                        ctl.Advance();
                        if (!__all_sync(0xffffffffu, WaitBarA(&misc.BarFull[slot], (g / HSTAGES) & 1, abortFlag))) {
                            fail(kDevTimeoutTma);
                            break;
                        }
                    }
                    if (!first && !__all_sync(0xffffffffu, WaitBarSleep<20>(&misc.BarP[h], (it - 1) & 1, abortFlag))) {
                        fail(kDevTimeoutMma);
                        break;
                    }
                    if (!__all_sync(0xffffffffu, takeTurn(2 * block + h))) {
                        fail(kDevTimeoutMma);
                        break;
                    }
                    TcFenceAfter();
                    if (ElectOne()) {
                        if (!first) {
                            issueOutputs(prevSlot, h);
                            MmaCommit(&misc.BarEmpty[prevSlot]);
                        }
                        if (more) {
                            issueScores(slot, h);
                            MmaCommit(&misc.BarS[h]);
                            if (!ctl.Valid) {
                                MmaCommit(&misc.BarREmpty);
                            }
                        } else {
                            MmaCommit(&misc.BarOut);
                        }
                    }
                    passTurn(2 * block + h);
                    ++block;
                    if (!more) {
                        break;
                    }
                    ++it;
                }
            }
            __syncwarp();
        }
        __syncwarp();
    } else {
        // ---------------------------------------------------------------- arithmetic warps
        const int quarter = tid >> 7;          // 16-column block of each 64-column half
        const int r = tid & (TILE_ROWS - 1);
        const uint32_t tLane = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        const float g = p.GlobalScale ? *p.GlobalScale : 1.0f;
        const float cg = p.C * g;
        const float dsMult = cg * kLog2;
        int rowTile = 0, head = 0, row = 0;
        TTileIter cur;
        // per-row constants.  dQ pass: the row is a query (scale sq, lse, delta); dK/dV pass: the row is a key (sk, sv)
        // (kept as loaded until an item's first tile, so that their latency passes behind the previous item's outputs)
        float rowScale = 0, rowLse = 0, rowOther = 0;
        float rowMult = 0;
        int spanS = 1, spanF = 0, spanRound = -1;
        // the tile's 128 column factors are staged by the first 128 threads, one tile ahead, and worked on when they are staged
        float pfA = 0, pfT = 0, pfB = 0;
        auto fetchCols = [&](int c0) {
            const int c = c0 + tid;
            const bool ok = tid < TILE_ROWS && c < p.Rows;
            pfA = 0;
            pfT = 0;
            pfB = 0;
            if (ok) {
                if (!MODE_DKV) {
                    pfA = p.KScale.Row(head)[c];
                    pfB = p.VScale.Valid() ? p.VScale.Row(head)[c] : p.VVecScale;
                } else {
                    pfA = p.QScale.Valid() ? p.QScale.Row(head)[c] : p.QkVecScale;
                    pfT = p.Lse.Row(head)[c];
                    pfB = p.DScale.Row(head)[c];
                }
            }
        };
        auto fetchSpans = [&]() {
            spanS = 1;
            spanF = 0;
            const tsa_span_group *gp = (r < 64) ? cur.G0 : cur.G1;
            const int n = (r < 64) ? cur.N0 : cur.N1;
            if (cur.Round < n) {
                spanS = gp[cur.Round].SpanStart[r & 63];
                spanF = gp[cur.Round].SpanFinish[r & 63];
            }
            spanRound = cur.Round;
        };
        // clears this thread's quarter of the output accumulators: every output product accumulates
        auto clearOutputs = [&]() {
            uint32_t zero[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                zero[k] = 0;
            }
#pragma unroll
            for (int o = 0; o < OUTPUTS; ++o) {
#pragma unroll
                for (int c = 0; c < QUARTER_D; c += 8) {
                    TmemSt8(tLane + BWD_OUT_COL + o * D + quarter * QUARTER_D + c, zero);
                }
            }
            TmemWaitSt();
            TcFenceBefore();
        };
        bool failed = false;
        // The next work item into (rowTile, head, cur); rowTile < 0: none.  False, in all threads alike, when a wait has run out somewhere: the arithmetic threads
        // leave together, none of them waits alone at a named barrier.
        auto takeItem = [&](int n) {
            const bool ok = WaitBarA(&misc.ItemFull[n & 1], (n >> 1) & 1, abortFlag);
            rowTile = misc.Item[n & 1].RowTile;
            head = misc.Item[n & 1].Head;
            cur = misc.Item[n & 1].First;
            if (BarRedOr(BAR_ARITH, BWD_ARITH_THREADS, failed || !ok)) {
                return false;
            }
            if (lane == 0) {
                MbarArrive(&misc.ItemEmpty[n & 1]);
            }
            return true;
        };
        auto setUp = [&]() {
            row = rowTile * TILE_ROWS + r;
            rowScale = 0;
            rowLse = 0;
            rowOther = 0;
            if (row < p.Rows) {
                if (!MODE_DKV) {
                    rowScale = p.QScale.Valid() ? p.QScale.Row(head)[row] : p.QkVecScale;
                    rowLse = p.Lse.Row(head)[row];
                    rowOther = p.DScale.Row(head)[row];
                } else {
                    rowScale = p.KScale.Row(head)[row];
                    rowOther = p.VScale.Valid() ? p.VScale.Row(head)[row] : p.VVecScale;
                }
            }
            if (cur.Valid) {
                fetchCols(cur.J0);
                fetchSpans();
            }
        };
        int it = 0, outCount = 0; // tiles, items with tiles
        bool alive = takeItem(0);
        if (alive && rowTile >= 0) {
            setUp();
            clearOutputs();
        }
        for (int n = 1; alive && rowTile >= 0; ++n) {
            const bool hasTiles = cur.Valid;
            rowMult = rowScale * cg;
            rowOther *= MODE_DKV ? dsMult : -dsMult;
            while (cur.Valid) {
                if (cur.Round != spanRound) {
                    fetchSpans();
                }
                const int buf = it & 1;
                if (tid < TILE_ROWS) {
                    misc.ColA[buf][tid] = pfA;
                    misc.ColT[buf][tid] = MODE_DKV ? -pfT - p.Slope * (float)tid : p.Slope * (float)tid;
                    misc.ColB[buf][tid] = MODE_DKV ? -pfB * dsMult : pfB * dsMult;
                    __syncwarp();
                    if (lane == 0) {
                        MbarArrive(&misc.ColFull[buf]);
                    }
                }
                const int c0 = cur.J0;
                const int ls = spanS - c0, lf = min(spanF, p.Rows - 1) - c0; // span in tile-local columns
                const bool rowFull = ls <= 0 && lf >= TILE_ROWS - 1;
                const bool warpMasked = !__all_sync(0xffffffffu, rowFull);
                // The staged columns, double buffered: a warp that stages tile t + 2 has seen the scores of tile t + 1's second half, and
                // those were asked for when all 16 warps had handed over tile t.  (A barrier of the 512 threads per tile kept the warps in
                // step.)  A thread whose wait fails goes to the threads' next common barrier, where they leave together.
                if (!__all_sync(0xffffffffu, !failed && WaitBarA<true>(&misc.ColFull[buf], (it >> 1) & 1, abortFlag, p.WaitCycles))) {
                    failed = true;
                    *(volatile int *)&misc.Abort = 1;
                    if (p.Status) {
                        atomicOr(p.Status, kDevTimeoutMma);
                    }
                    break;
                }
                {
                    TTileIter nxt = cur;
                    nxt.Advance();
                    if (nxt.Valid) {
                        fetchCols(nxt.J0);
                    }
                }
                // exponent = u * rowMult + (ColT + rowConst):  dQ: ALiBi + rowOff - lse_i;  dK/dV: -lse_i - ALiBi with the sign of the
                // transposed tile
                const float2 rowMult2 = make_float2(rowMult, rowMult), rowOther2 = make_float2(rowOther, rowOther);
                const float rowOff = -p.Slope * (float)(row - c0);
                const float rowConst = MODE_DKV ? -rowOff : rowOff - rowLse;
                const float2 rowConst2 = make_float2(rowConst, rowConst);
#pragma unroll 1
                for (int h = 0; h < 2; ++h) {
                    if (!WaitBarA(&misc.BarS[h], it & 1, abortFlag)) {
                        failed = true;
                        *(volatile int *)&misc.Abort = 1;
                        if (p.Status) {
                            atomicOr(p.Status, kDevTimeoutMma);
                        }
                        break; // to the next barrier of the arithmetic threads
                    }
                    TcFenceAfter();
                    const int cb = h * 64 + quarter * 16; // first tile column of this thread's block in the half
                    // span clipped to this block, block-local: (unsigned)(c - lsQ) <= spanW  <=>  inside the span
                    const int lsC = max(ls, cb), lfC = min(lf, cb + 15);
                    const bool rowEmpty = lsC > lfC;
                    const int lsQ = lsC - cb;
                    const unsigned spanW = rowEmpty ? 0u : (unsigned)(lfC - lsC);
                    uint32_t a1[8], a2[8];
                    // The arithmetic of a half's 16 columns, with and without the mask: as one piece of code every pair of columns carried
                    // six instructions that only tiles at the mask's edge need.
                    auto weigh = [&](auto maskedTag) {
                        constexpr bool MASKED = decltype(maskedTag)::value;
                        float2 s[8], d[8];
                        TmemLd16x2Pairs(tLane + BWD_S_COL + cb, tLane + BWD_DP_COL + cb, s, d);
                        const float4 *A4 = reinterpret_cast<const float4 *>(misc.ColA[buf] + cb);
                        const float4 *T4 = reinterpret_cast<const float4 *>(misc.ColT[buf] + cb);
                        const float4 *B4 = reinterpret_cast<const float4 *>(misc.ColB[buf] + cb);
#pragma unroll
                        for (int c = 0; c < 16; c += 4) {
                            const float4 a4 = A4[c >> 2], t4 = T4[c >> 2], b4 = B4[c >> 2];
#pragma unroll
                            for (int k = 0; k < 2; ++k) {
                                const int i = (c >> 1) + k;
                                const float2 ca = k ? make_float2(a4.z, a4.w) : make_float2(a4.x, a4.y);
                                const float2 ct = k ? make_float2(t4.z, t4.w) : make_float2(t4.x, t4.y);
                                const float2 cbv = k ? make_float2(b4.z, b4.w) : make_float2(b4.x, b4.y);
                                const float2 u = __fmul2_rn(s[i], ca);
                                const float2 e = __ffma2_rn(u, rowMult2, __fadd2_rn(ct, rowConst2));
                                float2 pij = FastExp2Pair(e);
                                if (MASKED) {
                                    pij.x = (!rowEmpty && (unsigned)(c + 2 * k - lsQ) <= spanW) ? pij.x : 0.0f;
                                    pij.y = (!rowEmpty && (unsigned)(c + 2 * k + 1 - lsQ) <= spanW) ? pij.y : 0.0f;
                                }
                                const float2 dpv = MODE_DKV ? __ffma2_rn(d[i], rowOther2, cbv) : __ffma2_rn(d[i], cbv, rowOther2);
                                const float2 ds = __fmul2_rn(__fmul2_rn(pij, dpv), ca);
                                a1[i] = PackBf16x2(ds.x, ds.y);
                                a2[i] = PackBf16x2(pij.x, pij.y);
                            }
                        }
                    };
                    if (!warpMasked) {
                        weigh(std::false_type());
                    } else if (__any_sync(0xffffffffu, !rowEmpty)) {
                        weigh(std::true_type());
                    } else {
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            a1[k] = 0;
                            a2[k] = 0;
                        }
                    }
                    // 16 bf16 values = 8 columns, written over the first half of the 16 columns this thread has just read
                    TmemSt8(tLane + BWD_S_COL + cb, a1);
                    if (MODE_DKV) {
                        TmemSt8(tLane + BWD_DP_COL + cb, a2);
                    }
                    TmemWaitSt();
                    TcFenceBefore();
                    __syncwarp();
                    if (lane == 0) {
                        MbarArrive(&misc.BarP[h]);
                    }
                }
                cur.Advance();
                ++it;
            }

            // The next item's spans, row constants and first column factors are looked up while this one's last output products run.
            const int doneRow = row, doneHead = head;
            alive = takeItem(n);
            if (!alive) {
                break;
            }
            if (rowTile >= 0) {
                setUp();
            }
            if (hasTiles) {
                if (!__all_sync(0xffffffffu, WaitBarA(&misc.BarOut, outCount & 1, abortFlag))) {
                    failed = true; // carried to the next item's barrier; without one the thread just leaves
                    *(volatile int *)&misc.Abort = 1;
                    if (p.Status) {
                        atomicOr(p.Status, kDevTimeoutMma);
                    }
                    continue;
                }
                ++outCount;
                TcFenceAfter();
            }
            // Outputs straight from the registers, 32 bytes (a whole sector) per store where the rows allow it: a thread holds a quarter
            // of one row.  The stores drain while the next item's score products run.
            const int esz = (p.GradDtype == TSA_F32) ? 4 : 2;
#pragma unroll
            for (int o = 0; o < OUTPUTS; ++o) {
                uint32_t v[QUARTER_D];
                if (hasTiles) {
                    if (QUARTER_D == 32) {
                        TmemLd32(tLane + BWD_OUT_COL + o * D + quarter * QUARTER_D, v);
                    } else {
                        TmemLd16(tLane + BWD_OUT_COL + o * D + quarter * QUARTER_D, v);
                    }
                    TmemWaitLd();
                } else {
#pragma unroll
                    for (int c = 0; c < QUARTER_D; ++c) {
                        v[c] = 0;
                    }
                }
                if (doneRow < p.Rows) {
                    const P2D<char> &outp = (o == 0) ? p.Out1 : p.Out2;
                    char *dst = outp.Row(doneRow) + (size_t)(doneHead * D + quarter * QUARTER_D) * esz;
                    auto put = [&](const uint32_t *w) { // 32 bytes
                        if (p.WideStores) {
                            StGlobal256(dst, w);
                        } else {
                            reinterpret_cast<uint4 *>(dst)[0] = make_uint4(w[0], w[1], w[2], w[3]);
                            reinterpret_cast<uint4 *>(dst)[1] = make_uint4(w[4], w[5], w[6], w[7]);
                        }
                        dst += 32;
                    };
                    if (p.GradDtype == TSA_F32) {
#pragma unroll
                        for (int c = 0; c < QUARTER_D; c += 8) {
                            uint32_t w[8];
#pragma unroll
                            for (int k = 0; k < 8; ++k) {
                                w[k] = __float_as_uint(__uint_as_float(v[c + k]) * p.GradMult);
                            }
                            put(w);
                        }
                    } else {
#pragma unroll
                        for (int c = 0; c < QUARTER_D; c += 16) {
                            uint32_t w[8];
#pragma unroll
                            for (int k = 0; k < 8; ++k) {
                                const float a = __uint_as_float(v[c + 2 * k]) * p.GradMult, b = __uint_as_float(v[c + 2 * k + 1]) * p.GradMult;
                                w[k] = (p.GradDtype == TSA_BF16) ? PackBf16x2(a, b) : PackHalf2(a, b);
                            }
                            put(w);
                        }
                    }
                }
            }
            if (hasTiles && rowTile >= 0) {
                clearOutputs();
            }
        }
    }
    if (MODE_DKV) {
        PdlWait();
    }
    TcFenceBefore();
    __syncthreads();
    if (warp == BWD_CTRL_WARP) {
        TmemDealloc(tmem, BWD_TMEM_COLS);
    }
}

// ---- widening of the stored vectors to bf16 ------------------------------------------------------------
// src: [rows][cols] of i8 / e4m3 / f16 / bf16 / f32 -> dst bf16 [rows][cols] (dense); 8 elements per thread
__global__ void __launch_bounds__(256) ToBf16Kernel(int srcDtype, P2D<char> src, int rows, int cols, __nv_bfloat16 *dst)
{
    PdlTrigger();
    PdlWait();
    const long long groups = (long long)rows * (cols / 8);
    for (long long gidx = blockIdx.x * (long long)blockDim.x + threadIdx.x; gidx < groups; gidx += (long long)gridDim.x * blockDim.x) {
        const int rowIdx = (int)(gidx / (cols / 8));
        const int c0 = (int)(gidx - (long long)rowIdx * (cols / 8)) * 8;
        const void *rowp = src.Row(rowIdx);
        uint32_t w[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            w[k] = PackBf16x2(LoadAsFloat(rowp, c0 + 2 * k, srcDtype), LoadAsFloat(rowp, c0 + 2 * k + 1, srcDtype));
        }
        *reinterpret_cast<uint4 *>(dst + (size_t)rowIdx * cols + c0) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// Q, K and V in one launch when all three are 8-bit with 16-byte aligned rows: blockIdx.y picks the matrix, a thread
// widens 16 elements (one 16-byte load, two 16-byte stores)
struct TWiden3 {
    const char *Src[3];
    int Stride[3];
    int Dtype[3];
    __nv_bfloat16 *Dst[3];
    int *Counters; // of the backward kernels that follow: set to zero
};

__device__ __forceinline__ uint32_t Widen2(uint32_t w, int shift, int dtype)
{
    if (dtype == TSA_I8) {
        // int8 -> f32 without a conversion instruction: the byte, biased by 128, becomes the low mantissa bits of 2^23
        // (ulp 1), and 2^23 + 128 is subtracted again; exact
        const uint32_t biased = w ^ 0x80808080u;
        const float a = __uint_as_float(__byte_perm(biased, 0x4B000000u, shift == 0 ? 0x7440 : 0x7442)) - 8388736.0f;
        const float b = __uint_as_float(__byte_perm(biased, 0x4B000000u, shift == 0 ? 0x7441 : 0x7443)) - 8388736.0f;
        return PackBf16x2(a, b);
    }
    return PackBf16x2(E4M3ToFloat((uint8_t)(w >> shift)), E4M3ToFloat((uint8_t)(w >> (shift + 8))));
}

__global__ void __launch_bounds__(256) Widen8x3Kernel(TWiden3 t, int rows, int cols)
{
    PdlTrigger();
    PdlWait();
    const int m = blockIdx.y;
    if (blockIdx.x == 0 && m == 0 && threadIdx.x < 2) {
        t.Counters[threadIdx.x] = 0;
    }
    const char *src = t.Src[m];
    const int stride = t.Stride[m], dtype = t.Dtype[m];
    __nv_bfloat16 *dst = t.Dst[m];
    const int perRow = cols / 16;
    const long long groups = (long long)rows * perRow;
    const long long step = (long long)gridDim.x * blockDim.x;
    // four independent 16-byte loads in flight per thread
    for (long long g0 = blockIdx.x * (long long)blockDim.x + threadIdx.x; g0 < groups; g0 += 4 * step) {
        uint4 in[4];
        int rowIdx[4], c0[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const long long gidx = g0 + u * step;
            rowIdx[u] = (int)(gidx / perRow);
            c0[u] = (int)(gidx - (long long)rowIdx[u] * perRow) * 16;
            if (gidx < groups) {
                in[u] = __ldg(reinterpret_cast<const uint4 *>(src + (size_t)rowIdx[u] * stride + c0[u]));
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (g0 + u * step < groups) {
                const uint32_t w[4] = {in[u].x, in[u].y, in[u].z, in[u].w};
                uint32_t o[8];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    o[2 * k] = Widen2(w[k], 0, dtype);
                    o[2 * k + 1] = Widen2(w[k], 16, dtype);
                }
                // one 32-byte store: a whole sector per thread (the workspace is 256-byte aligned, cols a multiple of 16)
                StGlobal256(dst + (size_t)rowIdx[u] * cols + c0[u], o);
            }
        }
    }
}

// ---- host side ------------------------------------------------------------------------------------------
bool Sm100BwdSupports(const tsa_att_cfg *cfg, int headCount)
{
    if (cfg->flags & TSA_FLAG_FORCE_GENERIC) {
        return false;
    }
    if (cfg->head_dim_qk != cfg->head_dim_v || (cfg->head_dim_qk != 64 && cfg->head_dim_qk != 128)) {
        return false;
    }
    return headCount > 0;
}

size_t Sm100BwdWorkspaceBytes(int headCount, int headDim, int rows)
{
    const size_t mat = ((size_t)rows * headCount * headDim * 2 + 255) / 256 * 256;
    return 256 + 4 * mat; // work-item counters of the two passes; Q, K, V, dO as bf16
}

template <int D, bool MODE_DKV>
static int LaunchBwdT(const CUtensorMap &r1, const CUtensorMap &r2, const CUtensorMap &c1, const CUtensorMap &c2, TBwdParams bp,
    int rowTiles, cudaStream_t stream)
{
    auto kern = BwdSm100Kernel<D, MODE_DKV>;
    const int smemBytes = TBwdSmem<D>::TOTAL;
    int rc = CheckCuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smemBytes), "cudaFuncSetAttribute(backward)");
    if (rc != TSA_OK) {
        return rc;
    }
    int dev = 0, sms = 0;
    rc = CheckCuda(cudaGetDevice(&dev), "cudaGetDevice");
    if (rc == TSA_OK) {
        rc = CheckCuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "cudaDeviceGetAttribute");
    }
    if (rc != TSA_OK) {
        return rc;
    }
    bp.Items = rowTiles * bp.HeadCount;
    void *args[] = {(void *)&r1, (void *)&r2, (void *)&c1, (void *)&c2, &bp};
    return CheckCuda(LaunchPdl((const void *)kern, dim3(bp.Items < sms ? bp.Items : sms), dim3(BWD_THREADS), smemBytes, stream, args), "tcgen05 backward launch");
}

int LaunchSm100Bwd(const tsa_att_cfg *cfg, const TGenParams &p, tsa_ptr2d qk, tsa_ptr2d qv, tsa_ptr2d v, tsa_ptr2d dOut,
    int lenAttTiles, void *workspace, int *statusWord, cudaStream_t stream)
{
    const int D = cfg->head_dim_qk;
    const int rows = p.Len;
    const int cols = p.HeadCount * D;
    const size_t mat = ((size_t)rows * cols * 2 + 255) / 256 * 256;
    int *counters = (int *)workspace;
    workspace = (char *)workspace + 256;
    __nv_bfloat16 *qb = (__nv_bfloat16 *)workspace;
    __nv_bfloat16 *kb = (__nv_bfloat16 *)((char *)workspace + mat);
    __nv_bfloat16 *vb = (__nv_bfloat16 *)((char *)workspace + 2 * mat);
    __nv_bfloat16 *dob = (__nv_bfloat16 *)((char *)workspace + 3 * mat);
    const long long groups = (long long)rows * (cols / 8);
    const int blocks = (int)((groups + 255) / 256 < 148 * 16 ? (groups + 255) / 256 : 148 * 16);
    auto aligned16 = [](const tsa_ptr2d &a) { return (uintptr_t)a.data % 16 == 0 && a.stride_bytes % 16 == 0; };
    if (cols % 16 == 0 && aligned16(qk) && aligned16(qv) && aligned16(v)) {
        TWiden3 t;
        const tsa_ptr2d *srcs[3] = {&qk, &qv, &v};
        __nv_bfloat16 *dsts[3] = {qb, kb, vb};
        for (int m = 0; m < 3; ++m) {
            t.Src[m] = (const char *)srcs[m]->data;
            t.Stride[m] = srcs[m]->stride_bytes;
            t.Dtype[m] = (m < 2) ? cfg->qk_dtype : cfg->v_dtype;
            t.Dst[m] = dsts[m];
        }
        const long long g16 = (long long)rows * (cols / 16);
        const int b16 = (int)((g16 + 255) / 256 < 148 * 8 ? (g16 + 255) / 256 : 148 * 8);
        t.Counters = counters;
        int r = rows, c = cols;
        void *args[] = {&t, &r, &c};
        const int rc = CheckCuda(LaunchPdl((const void *)Widen8x3Kernel, dim3(b16, 3), dim3(256), 0, stream, args), "bf16 widening launch");
        if (rc != TSA_OK) {
            return rc;
        }
    } else {
        const int rc = CheckCuda(cudaMemsetAsync(counters, 0, 256, stream), "clearing the backward counters");
        if (rc != TSA_OK) {
            return rc;
        }
        LaunchPdlArgs(ToBf16Kernel, dim3(blocks), dim3(256), 0, stream, cfg->qk_dtype, P2D<char>(qk), rows, cols, qb);
        LaunchPdlArgs(ToBf16Kernel, dim3(blocks), dim3(256), 0, stream, cfg->qk_dtype, P2D<char>(qv), rows, cols, kb);
        LaunchPdlArgs(ToBf16Kernel, dim3(blocks), dim3(256), 0, stream, cfg->v_dtype, P2D<char>(v), rows, cols, vb);
    }
    // dO that already is bf16 in a TMA-compatible layout is read where it lies
    const bool dOutInPlace = cfg->grad_dtype == TSA_BF16 && (uintptr_t)dOut.data % 16 == 0 && dOut.stride_bytes % 16 == 0 && dOut.xsize >= cols;
    if (!dOutInPlace) {
        LaunchPdlArgs(ToBf16Kernel, dim3(blocks), dim3(256), 0, stream, cfg->grad_dtype, P2D<char>(dOut), rows, cols, dob);
    }
    int rc = CheckCuda(cudaGetLastError(), "bf16 widening launch");
    if (rc != TSA_OK) {
        return rc;
    }
    auto mapOf = [&](CUtensorMap *m, __nv_bfloat16 *ptr, const char *what) {
        tsa_ptr2d a = {ptr, cols * 2, cols, rows};
        return MakeTileMapEx(m, a, 2, 64, 64, what);
    };
    CUtensorMap mq, mk, mv, mdo;
    rc = mapOf(&mq, qb, "q bf16");
    if (rc == TSA_OK) {
        rc = mapOf(&mk, kb, "k bf16");
    }
    if (rc == TSA_OK) {
        rc = mapOf(&mv, vb, "v bf16");
    }
    if (rc == TSA_OK) {
        if (dOutInPlace) {
            tsa_ptr2d a = {dOut.data, dOut.stride_bytes, cols, rows};
            rc = MakeTileMapEx(&mdo, a, 2, 64, 64, "dOut bf16 (in place)");
        } else {
            rc = mapOf(&mdo, dob, "dOut bf16");
        }
    }
    if (rc != TSA_OK) {
        return rc;
    }
    TBwdParams bp;
    bp.HeadCount = p.HeadCount;
    bp.Rows = rows;
    bp.LenAttTiles = lenAttTiles;
    bp.QScale = p.QScale;
    bp.KScale = p.KScale;
    bp.VScale = p.VScale;
    bp.QkVecScale = p.QkVecScale;
    bp.VVecScale = p.VVecScale;
    bp.Lse = p.Lse;
    bp.DScale = p.DScale;
    bp.GlobalScale = p.GlobalScale;
    bp.C = p.C;
    bp.Slope = p.Slope;
    bp.GradMult = p.GradMult;
    bp.GradDtype = p.GradDtype;
    bp.Status = statusWord;
    bp.WaitCycles = TestHooks().WaitCycles > 0 ? TestHooks().WaitCycles : WAIT_CYCLES;
    bp.WithholdTile = TestHooks().WithholdTile;
    const int rowTiles = (lenAttTiles + 1) / 2;
    // dQ pass: rows = queries
    bp.Spans = p.Spans;
    bp.SpanPtr = p.SpanPtr;
    bp.Out1 = p.DQ;
    bp.Out2 = p.DQ;
    auto wide = [](const P2D<char> &a) { return (((uintptr_t)a.Data | (uintptr_t)a.Stride) & 31) == 0; };
    bp.WideStores = wide(p.DQ);
    bp.Ascending = 0;
    bp.Counter = counters;
    rc = (D == 128) ? LaunchBwdT<128, false>(mq, mdo, mk, mv, bp, rowTiles, stream) : LaunchBwdT<64, false>(mq, mdo, mk, mv, bp, rowTiles, stream);
    if (rc != TSA_OK) {
        return rc;
    }
    // dK / dV pass: rows = keys, columns from the transposed spans
    bp.Spans = p.RevSpans;
    bp.SpanPtr = p.RevSpanPtr;
    bp.Out1 = p.DK;
    bp.Out2 = p.DV;
    bp.WideStores = wide(p.DK) && wide(p.DV);
    bp.Ascending = 1;
    bp.Counter = counters + 1;
    return (D == 128) ? LaunchBwdT<128, true>(mk, mv, mq, mdo, bp, rowTiles, stream) : LaunchBwdT<64, true>(mk, mv, mq, mdo, bp, rowTiles, stream);
}

} // namespace tsa
