// Inner loop of the KV-cache attention, shared by the decode kernel and the persistent inference step: one warp streams a range
// of tokens of one sequence for 32 / (D / 16) heads.
#pragma once
#include "tsa_common.cuh"

namespace tsa {

__device__ __forceinline__ void KeyRange(int ctxLen, int window, int *j0, int *j1)
{
    int cur = ctxLen - 1;
    if (window == 0) {
        *j0 = cur;
        *j1 = cur + 1;
    } else {
        *j0 = max(0, cur - window);
        *j1 = cur;
    }
}

template <bool F16>
struct TScaleOf {
    typedef __half T;
};
template <>
struct TScaleOf<false> {
    typedef float T;
};
// COHERENT: the cache rows may have been written by this kernel (L2 loads instead of the read-only path)
template <bool COHERENT>
__device__ __forceinline__ float LoadScaleT(const __half *p)
{
    return __half2float(COHERENT ? __ldcg(p) : __ldg(p));
}
template <bool COHERENT>
__device__ __forceinline__ float LoadScaleT(const float *p)
{
    return COHERENT ? __ldcg(p) : __ldg(p);
}
template <bool COHERENT>
__device__ __forceinline__ int4 LoadRow(const int4 *p)
{
    return COHERENT ? __ldcg(p) : __ldg(p);
}
// two 16-bit x 8-bit products added to c: a = (w0 | w1 << 16) unsigned, b bytes signed; lo takes bytes 0 and 1 of b, hi bytes 2 and 3
__device__ __forceinline__ int Dp2aLoUS(uint32_t a, uint32_t b, int c)
{
    int d;
    asm("dp2a.lo.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ int Dp2aHiUS(uint32_t a, uint32_t b, int c)
{
    int d;
    asm("dp2a.hi.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

// Tokens [tBeg, tEnd) for this lane's 16-byte slice of its head: kp, vp, ksp, vsp point at token tBeg, qv is the query's slice.
// Keeps UNROLL tokens of K and V in flight; online softmax in (m, l, acc), batch after batch.  The warp runs `batches` of them, enough
// for every lane; a lane that has no tokens left repeats its last one (token tEnd - 1 has to be readable) with weight zero, which changes
// none of its sums.  A lane that never had one keeps m = -1e30, and its l and acc mean nothing.
template <int D, int UNROLL, bool COHERENT, class TScale>
__device__ __forceinline__ void AttendTokens(const int4 qv, float logitMult, float slope, int cur, const int4 *kp, const int4 *vp, const TScale *ksp,
    const TScale *vsp, int H, int tBeg, int tEnd, int batches, float &m, float &l, float (&acc)[16])
{
    constexpr int LPH = D / 16;     // lanes per head
    const int rowInt4 = H * D / 16; // int4 words per token row
    for (int tBase = tBeg; batches > 0; --batches, tBase += UNROLL) {
        int4 kv[UNROLL], vv[UNROLL];
        float ks[UNROLL], vs[UNROLL];
        const int cnt = tEnd - tBase; // tokens left
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            const int tt = min(u, cnt - 1);
            kv[u] = LoadRow<COHERENT>(kp + tt * rowInt4);
            vv[u] = LoadRow<COHERENT>(vp + tt * rowInt4);
            ks[u] = LoadScaleT<COHERENT>(ksp + tt * H);
            vs[u] = LoadScaleT<COHERENT>(vsp + tt * H);
        }
        kp += UNROLL * rowInt4;
        vp += UNROLL * rowInt4;
        ksp += UNROLL * H;
        vsp += UNROLL * H;
        float z[UNROLL];
        float cm = m;
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            int dot = __dp4a(qv.x, kv[u].x, 0);
            dot = __dp4a(qv.y, kv[u].y, dot);
            dot = __dp4a(qv.z, kv[u].z, dot);
            dot = __dp4a(qv.w, kv[u].w, dot);
#pragma unroll
            for (int o = LPH / 2; o > 0; o >>= 1) {
                dot += __shfl_xor_sync(0xffffffffu, dot, o);
            }
            // same association as the reference: ((dot * kScale) * attDotScale) * qScale - slope * dist
            const float zz = (float)dot * ks[u] * logitMult - slope * (float)(cur - (tBase + u));
            z[u] = (u < cnt) ? zz : -1e30f;
            cm = fmaxf(cm, z[u]);
        }
        if (cm != m) {
            const float corr = exp2f(m - cm);
            m = cm;
            l *= corr;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                acc[i] *= corr;
            }
        }
        // weights times value scales of the batch as 16-bit integers relative to the batch maximum (relative error of a
        // weight at most 2^-17 of the largest one), so that the 8 x 16 byte products run as two-token integer dot
        // products (dp2a) instead of a convert and a multiply-add per byte; one float update per batch
        float wv[UNROLL];
        float bmax = 0;
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            const float w = exp2f(z[u] - m);
            l += w;
            wv[u] = w * vs[u];
            bmax = fmaxf(bmax, wv[u]);
        }
        const float qScale = bmax > 0 ? 65535.0f / bmax : 0.0f;
        int iacc[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            iacc[i] = 0;
        }
#pragma unroll
        for (int u = 0; u < UNROLL; u += 2) {
            const uint32_t wp = __float2uint_rn(wv[u] * qScale) | (__float2uint_rn(wv[u + 1] * qScale) << 16);
            const uint32_t w0[4] = {(uint32_t)vv[u].x, (uint32_t)vv[u].y, (uint32_t)vv[u].z, (uint32_t)vv[u].w};
            const uint32_t w1[4] = {(uint32_t)vv[u + 1].x, (uint32_t)vv[u + 1].y, (uint32_t)vv[u + 1].z, (uint32_t)vv[u + 1].w};
#pragma unroll
            for (int wi = 0; wi < 4; ++wi) {
                // bytes (t0 b0, t1 b0, t0 b1, t1 b1) and (t0 b2, t1 b2, t0 b3, t1 b3)
                const uint32_t lo = __byte_perm(w0[wi], w1[wi], 0x5140);
                const uint32_t hi = __byte_perm(w0[wi], w1[wi], 0x7362);
                iacc[wi * 4 + 0] = Dp2aLoUS(wp, lo, iacc[wi * 4 + 0]);
                iacc[wi * 4 + 1] = Dp2aHiUS(wp, lo, iacc[wi * 4 + 1]);
                iacc[wi * 4 + 2] = Dp2aLoUS(wp, hi, iacc[wi * 4 + 2]);
                iacc[wi * 4 + 3] = Dp2aHiUS(wp, hi, iacc[wi * 4 + 3]);
            }
        }
        const float deq = bmax * (1.0f / 65535.0f);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            acc[i] = fmaf((float)iacc[i], deq, acc[i]);
        }
    }
}

} // namespace tsa
