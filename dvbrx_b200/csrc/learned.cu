/*
 * Learned (neural offset / scaled) min-sum: training kernels.
 *
 * The decoder is the plain layered decoder's schedule (layers in order,
 * wavefront steps inside levelled layers) with the check node's offset 1
 * replaced by a learned scale and offset per iteration t and check-degree
 * class k:
 *
 *     x_c   = clamp(P_v - m_c, -128, 127)            extrinsic input
 *     mu_c  = min(min_{c' != c} |x_c'|, 127)
 *     mag_c = max(beta[t][k] * mu_c - alpha[t][k], 0)
 *     m'_c  = sign_{c' != c}(x) * mag_c               (sign of 0 is +)
 *     P'_v  = clamp(x_c + m'_c, -128, 127)            posterior
 *     m_c  <- clamp(m'_c, -32, 31)                    stored message
 *
 * on the int8 decoder's scale (2 x LLR), with the same saturations as the
 * int8 decoder, in fp32.  The plain decoder is beta = 1, alpha = 1 (with
 * rounding).  The loss is the binary cross-entropy of the information bits
 * after every iteration: sum_t sum_v softplus(-(1 - 2 b_v) P_v / 2).
 *
 * One CTA per frame, thread j holding check j of every layer; posteriors in
 * global memory, a check's messages as one 16-byte record (the two magnitudes,
 * the outgoing signs, the links that hold the minimum), exact in fp32.  Degrees
 * are compiled apart, so a check's links stay in registers.
 *
 * Forward (k_learned_fwd): when training, every iteration leaves its extrinsic
 * inputs (one float per link) and its information posteriors.
 *
 * Backward (k_learned_bwd): for t = T-1 .. 0 it adds the iteration's loss
 * gradient, from the saved posteriors, then walks the layers and levels in
 * reverse from the saved extrinsic inputs, which give back the check node: the
 * gradient of a check node's outputs goes to its inputs through the straight
 * path (P' = x + m'), the scale and offset, and the minimum (the argmin link
 * receives d mag / d mu; the sign is piecewise constant); saturated clamps
 * pass no gradient.
 */
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "codes.h"
#include "learned.h"

namespace drxg {

constexpr int kLT = 384;
constexpr int kQCl = 360;

__device__ __forceinline__ float clampf(float v, float lo, float hi) { return fminf(fmaxf(v, lo), hi); }
__device__ __forceinline__ float softplus(float u) { return fmaxf(u, 0.0f) + log1pf(expf(-fabsf(u))); }
__device__ __forceinline__ float sigmoid(float u) { return 1.0f / (1.0f + expf(-u)); }

constexpr int kSharedMax = 12;               /* shared links of a layer at most: slots 2 .. 13 (codes.cpp puts them first) */
constexpr int kSharedEnd = 2 + kSharedMax;

/* The code's link tables, staged in shared memory: an entry (360 g - a, a) as
 * (byte offset of group g's first posterior, -4 a). */
struct LTables {
    const uint2* ent;
    const uint16_t* eoff;
    const uint8_t* nlev;
    const uint8_t* first; /* per entry: the layer's first entry of the same group */
    float* pass;          /* the shared links' values from level to level: [first][360] */
};

__device__ LTables stage_tables(const DevCode& c, char* smem)
{
    float* pass = (float*)smem;
    uint2* ent = (uint2*)(pass + kQCl * kSharedMax);
    uint16_t* eoff = (uint16_t*)(ent + c.nent);
    uint8_t* nlev = (uint8_t*)(eoff + c.q + 1);
    uint8_t* first = nlev + c.q;
    for (int i = threadIdx.x; i < c.q; i += blockDim.x)
        for (int e = c.eoff[i]; e < c.eoff[i + 1]; e++) {
            const int2 own = c.ent[e];
            int n = 0;
            while (c.ent[c.eoff[i] + n].x + c.ent[c.eoff[i] + n].y != own.x + own.y)
                n++;
            first[e] = (uint8_t)n;
        }
    for (int k = threadIdx.x; k < c.nent; k += blockDim.x) {
        const int2 e = c.ent[k];
        ent[k] = make_uint2(4u * (uint32_t)(e.x + e.y), 0u - 4u * (uint32_t)e.y);
    }
    for (int k = threadIdx.x; k <= c.q; k += blockDim.x)
        eoff[k] = c.eoff[k];
    for (int k = threadIdx.x; k < c.q; k += blockDim.x)
        nlev[k] = c.nlev[k];
    return LTables{ ent, eoff, nlev, first, pass };
}

/* Byte offset in a frame's posteriors of link `slot` of check (i, j): slot 0 =
 * parity, slot 1 = previous parity (absent for (0, 0)), 2.. = information bits
 * (ent: the layer's entries), bit (j - a) mod 360 of the group. */
__device__ __forceinline__ uint32_t link_at(const DevCode& c, const uint2* ent, int i, int j, int slot)
{
    if (slot == 0)
        return 4u * (uint32_t)(c.K + kQCl * i + j);
    if (slot == 1)
        return 4u * (uint32_t)(i ? c.K + kQCl * (i - 1) + j : c.K + kQCl * (c.q - 1) + j - 1);
    const uint2 e = ent[slot - 2];
    const uint32_t u = 4u * (uint32_t)j + e.y;
    return e.x + __viaddmin_u32(u, 4u * kQCl, u);
}

/* Where a shared link's value passes from one level to the next: bit (j - a)
 * mod 360 of the group that the layer's entry `first` names. */
__device__ __forceinline__ float& pass_at(const LTables& tb, int e, int j)
{
    const uint32_t u = 4u * (uint32_t)j + tb.ent[e].y;
    return *(float*)((char*)(tb.pass + kQCl * tb.first[e]) + __viaddmin_u32(u, 4u * kQCl, u));
}

__device__ __forceinline__ float& at(float* base, uint32_t offset) { return *(float*)((char*)base + offset); }

constexpr uint32_t kSign = 0x80000000u;
__device__ __forceinline__ uint32_t bits_of(float x) { return __float_as_uint(x); }
/* magnitude with a sign bit */
__device__ __forceinline__ float signed_by(float mag, uint32_t sign) { return __uint_as_float(bits_of(mag) | (sign & kSign)); }

/* the two smallest of magnitudes a taken one after the other */
__device__ __forceinline__ void two_smallest(float& m0, float& m1, float a)
{
    m1 = fminf(m1, fmaxf(m0, a));
    m0 = fminf(m0, a);
}

constexpr float kNone = 1e30f;  /* above every magnitude */

/* Loss of the posteriors after an iteration (and a copy of them). */
__device__ float iteration_loss(const DevCode& c, const float* __restrict__ P, const LearnedParams& p, int f,
                                float* __restrict__ copy)
{
    const uint8_t* bits = p.bits + (size_t)f * p.bits_stride;
    float acc = 0.0f;
#pragma unroll 8
    for (int v = threadIdx.x; v < c.kldpc; v += kLT) {
        const float sb = ((bits[v >> 3] >> (7 - (v & 7))) & 1) ? -1.0f : 1.0f; /* +1 for a 0 bit */
        const float x = P[v];
        if (copy)
            __stcs(copy + v, x);
        acc += softplus(-sb * x * 0.5f);
    }
    return acc;
}

__device__ float block_sum(float v, float* red)
{
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    if ((threadIdx.x & 31) == 0)
        red[threadIdx.x >> 5] = v;
    __syncthreads();
    float r = 0.0f;
    if (threadIdx.x == 0)
        for (int w = 0; w < (int)(blockDim.x >> 5); w++)
            r += red[w];
    __syncthreads();
    return r;
}

__device__ void load_params(const LearnedParams& p, int t, float* sbeta, float* salpha)
{
    if ((int)threadIdx.x < p.nclass) {
        sbeta[threadIdx.x] = __half2float(p.beta[t * p.nclass + threadIdx.x]);
        salpha[threadIdx.x] = __half2float(p.alpha[t * p.nclass + threadIdx.x]);
    }
    __syncthreads();
}

/*
 * A layer runs in three parts, as in the int8 decoder: all checks load the
 * links that no earlier check of the layer writes and reduce those that no
 * other check shares; the wavefront levels then carry the shared links alone
 * (a message to one has the smallest magnitude of the unshared links and of the
 * other shared ones); a last part takes the shared links into the minimums and
 * writes everything else.  The magnitudes and signs are those of the node as a
 * whole, so the values do not depend on the split.  Shared links pass from
 * level to level in shared memory.
 *
 * Bound by the dependent steps of a frame's layers: one frame alone on an SM
 * takes 0.65 ms per iteration forward and backward, three or four 1.7 ms; DRAM
 * is under 20 %.  512 normal 2/3 frames, 20 iterations, loss and gradients:
 * 73.5 ms with the whole check node in every level step, 33.7 ms so.  (Extrinsic
 * inputs and message gradients fetched a layer ahead into shared memory: 34.6;
 * link addresses kept in registers: 42, by spills.)
 *
 * EXACT: every layer has DM links; otherwise up to DM, by a uniform predicate.
 */

/* resident CTAs per SM that a degree's registers are compiled for */
__host__ __device__ constexpr int fwd_ctas(int dm) { return dm <= 11 ? 3 : dm <= 22 ? 2 : 1; }
__host__ __device__ constexpr int bwd_ctas(int dm) { return dm <= 18 ? 2 : 1; }

template <int DM, bool EXACT>
__global__ void __launch_bounds__(kLT, fwd_ctas(DM)) k_learned_fwd(LearnedParams p)
{
    extern __shared__ __align__(16) char smem[];
    __shared__ float sbeta[kLearnedMaxClass], salpha[kLearnedMaxClass], red[kLT / 32];
    const DevCode c = *p.code;
    const LTables tb = stage_tables(c, smem);
    const int f = blockIdx.x, j = threadIdx.x;
    const bool active = j < kQCl;
    float* P = p.P + (size_t)f * c.N;
    uint4* M = p.M + (size_t)f * c.R;
    const __half* src = p.llr + (size_t)f * p.llr_stride;
    /* + 0: no negative zeros, so that a sign bit is a sign */
    for (int v = j; v < c.K; v += blockDim.x)
        P[v] = clampf(__half2float(src[v]), -128.0f, 127.0f) + 0.0f;
    for (int k = j; k < c.R; k += blockDim.x)
        P[c.K + kQCl * (k % c.q) + k / c.q] = clampf(__half2float(src[c.K + k]), -128.0f, 127.0f) + 0.0f;
    __syncthreads();
    for (int t = 0; t < p.iters; t++) {
        load_params(p, t, sbeta, salpha);
        float* X = p.Xck ? p.Xck + ((size_t)t * p.nframes + f) * p.DS * c.R + j : nullptr;
        uint4 rn = make_uint4(0, 0, 0, 0); /* records and levels one layer ahead; no messages at first */
        unsigned long long mn = 0;
        if (active) {
            if (t)
                rn = M[j];
            mn = __ldg(c.lmeta + j);
        }
        for (int i = 0; i < c.q; i++) {
            const uint4 rec = rn;
            const unsigned long long meta = mn;
            if (active && i + 1 < c.q) {
                if (t)
                    rn = M[kQCl * (i + 1) + j];
                mn = __ldg(c.lmeta + kQCl * (i + 1) + j);
            }
            const int e0 = tb.eoff[i];
            const uint2* ent = tb.ent + e0;
            const int D = EXACT ? DM : tb.eoff[i + 1] - e0 + 2, nl = tb.nlev[i];
            const bool pp = (i | j) != 0;
            auto on = [&](int k) { return (EXACT || k < D) && (k != 1 || pp); };
            const uint32_t late = (uint32_t)(meta >> 8) & 0xFFFFFFu, early = (uint32_t)(meta >> 32) & 0xFFFFFFu;
            const uint32_t shared = late | early;
            const int lev = (int)(meta & 0xFF);
            float raw[DM];
            auto load = [&](int k, float post) {
                const float mag = __uint_as_float((rec.w >> k) & 1u ? rec.y : rec.x);
                const float m = clampf(signed_by(mag, rec.z << (31 - k)), -32.0f, 31.0f); /* the link's old message */
                raw[k] = post - m;
            };
            auto input = [&](int k) { return clampf(raw[k], -128.0f, 127.0f); };
            float min0 = kNone, min1 = kNone;
            uint32_t par = 0; /* sign bit: the parity of the inputs' signs */
            auto take = [&](int k) {
                const float x = input(k);
                two_smallest(min0, min1, fabsf(x));
                par ^= bits_of(x);
            };
            float beta = 0.0f, alpha = 0.0f;
            auto magnitude = [&](float m) { return fmaxf(beta * fminf(m, 127.0f) - alpha, 0.0f); };
            if (active) {
                const int cl = p.cls[D - (pp ? 0 : 1)];
                beta = sbeta[cl];
                alpha = salpha[cl];
#pragma unroll
                for (int k = 0; k < DM; k++)
                    if (on(k) && !((late >> k) & 1u))
                        load(k, at(P, link_at(c, ent, i, j, k)));
#pragma unroll
                for (int k = 0; k < DM; k++)
                    if (on(k) && !((shared >> k) & 1u))
                        take(k);
            }
            if (nl > 1) {
                auto levels = [&](auto end) {
                    constexpr int KE = decltype(end)::value < DM ? decltype(end)::value : DM; /* shared slots are 2 .. KE - 1 */
                    for (int l = 0; l < nl; l++) {
                        if (active && lev == l) {
                            float s0 = kNone, s1 = kNone;
                            uint32_t sp = par;
#pragma unroll
                            for (int k = 2; k < KE; k++)
                                if (KE == 4 || ((shared >> k) & 1u)) {
                                    if ((late >> k) & 1u)
                                        load(k, pass_at(tb, e0 + k - 2, j));
                                    const float x = input(k);
                                    two_smallest(s0, s1, fabsf(x));
                                    sp ^= bits_of(x);
                                }
#pragma unroll
                            for (int k = 2; k < KE; k++)
                                if ((early >> k) & 1u) {
                                    const float x = input(k);
                                    const float m = magnitude(fminf(min0, fabsf(x) == s0 ? s1 : s0));
                                    pass_at(tb, e0 + k - 2, j) =
                                        clampf(x + signed_by(m, sp ^ bits_of(x)), -128.0f, 127.0f);
                                }
                        }
                        if (l + 1 < nl) /* nothing waits for the last level */
                            __syncthreads();
                    }
                    if (active) {
#pragma unroll
                        for (int k = 2; k < KE; k++)
                            if (KE == 4 || ((shared >> k) & 1u))
                                take(k);
                    }
                };
                /* the same for every check of the layer: two shared slots, up to four, more */
                const uint32_t any = __reduce_or_sync(0xFFFFFFFFu, shared);
                if (!(any >> 4))
                    levels(std::integral_constant<int, 4>());
                else if (!(any >> 6))
                    levels(std::integral_constant<int, 6>());
                else
                    levels(std::integral_constant<int, kSharedEnd>());
            }
            if (active) {
                const float mag0 = magnitude(min0), mag1 = magnitude(min1);
                uint32_t signs = 0, own = 0; /* of the outgoing messages; links that hold the minimum */
#pragma unroll
                for (int k = 0; k < DM; k++)
                    if (on(k)) {
                        const float x = input(k);
                        const bool is = fabsf(x) == min0;
                        const uint32_t sn = (par ^ bits_of(x)) & kSign;
                        const float m = signed_by(is ? mag1 : mag0, sn);
                        signs |= sn >> (31 - k);
                        own |= is ? 1u << k : 0u;
                        if (!((early >> k) & 1u))
                            at(P, link_at(c, ent, i, j, k)) = clampf(x + m, -128.0f, 127.0f);
                        if (X)
                            __stcs(X + (size_t)kQCl * (p.DS * i) + kQCl * k, raw[k]);
                    }
                M[kQCl * i + j] = make_uint4(bits_of(mag0), bits_of(mag1), signs, own);
            }
            __syncthreads();
        }
        float* copy = p.Pck ? p.Pck + ((size_t)t * p.nframes + f) * c.K : nullptr;
        const float l = block_sum(iteration_loss(c, P, p, f, copy), red);
        if (j == 0)
            atomicAdd(p.loss + t, l);
    }
    if (p.post)
        for (int v = j; v < c.kldpc; v += blockDim.x)
            p.post[(size_t)f * c.kldpc + v] = P[v];
}

/* The gradient runs the layers and levels backwards: a check's outputs that
 * later checks of the layer read (early) have their gradient from those
 * checks' levels, and earlier levels wait for the gradients of its inputs that
 * earlier checks wrote (late).  Everything else is summed before the first
 * level and written after the last. */
template <int DM, bool EXACT>
__global__ void __launch_bounds__(kLT, bwd_ctas(DM)) k_learned_bwd(LearnedParams p)
{
    extern __shared__ __align__(16) char smem[];
    __shared__ float sbeta[kLearnedMaxClass], salpha[kLearnedMaxClass];
    __shared__ double sdb[kLearnedMaxClass], sda[kLearnedMaxClass];
    const DevCode c = *p.code;
    const LTables tb = stage_tables(c, smem);
    const int f = blockIdx.x, j = threadIdx.x, lane = j & 31;
    const bool active = j < kQCl;
    const size_t E = (size_t)p.DS * c.R;
    float* gP = p.gP + (size_t)f * c.N;
    float* gM = p.gM + (size_t)f * E + j;
    const uint8_t* bits = p.bits + (size_t)f * p.bits_stride;
    for (int t = p.iters - 1; t >= 0; t--) {
        const bool lastit = t == p.iters - 1;
        if (j < kLearnedMaxClass)
            sdb[j] = sda[j] = 0.0;
        load_params(p, t, sbeta, salpha);
        /* the gradient of the iteration's loss */
        const float* P = p.Pck + ((size_t)t * p.nframes + f) * c.K;
        const float* X = p.Xck + ((size_t)t * p.nframes + f) * E + j;
        const float gscale = p.loss_scale * (p.loss_w ? p.loss_w[t] : 1.0f);
        auto gradient_of_loss = [&](int v) {
            const float sb = ((bits[v >> 3] >> (7 - (v & 7))) & 1) ? -1.0f : 1.0f;
            return gscale * (-sb * 0.5f) * sigmoid(-sb * __ldcs(P + v) * 0.5f);
        };
        if (lastit) {
#pragma unroll 8
            for (int v = j; v < c.N; v += kLT)
                gP[v] = v < c.kldpc ? gradient_of_loss(v) : 0.0f;
        } else {
#pragma unroll 8
            for (int v = j; v < c.kldpc; v += kLT)
                gP[v] += gradient_of_loss(v);
        }
        __syncthreads();
        double db = 0.0, da = 0.0; /* of the layers' class since the last flush */
        for (int i = c.q - 1; i >= 0; i--) {
            const int first = tb.eoff[i];
            const uint2* ent = tb.ent + first;
            const int D = EXACT ? DM : tb.eoff[i + 1] - first + 2, nl = tb.nlev[i];
            const bool pp = (i | j) != 0;
            auto on = [&](int k) { return (EXACT || k < D) && (k != 1 || pp); };
            const float* Xl = X + (size_t)kQCl * (p.DS * i);
            float* gMl = gM + (size_t)kQCl * (p.DS * i);
            float raw[DM], go[DM]; /* go: first the message's gradient, then the posterior's that passes */
            uint32_t early = 0, late = 0;
            int lev = 0;
            if (active) {
                const unsigned long long meta = __ldg(c.lmeta + kQCl * i + j);
                late = (uint32_t)(meta >> 8) & 0xFFFFFFu;
                early = (uint32_t)(meta >> 32) & 0xFFFFFFu;
                lev = (int)(meta & 0xFF);
#pragma unroll
                for (int k = 0; k < DM; k++)
                    if (on(k)) {
                        raw[k] = __ldcs(Xl + kQCl * k);
                        go[k] = lastit ? 0.0f : __ldcs(gMl + kQCl * k);
                    }
            }
            /* the node: minimums, the links that hold them (the first of equal ones), signs */
            float min0 = kNone, min1 = kNone;
            uint32_t neg = 0, e0 = 0, e1 = 0;
            auto input = [&](int k) { return clampf(raw[k], -128.0f, 127.0f); };
            if (active) {
#pragma unroll
                for (int k = 0; k < DM; k++)
                    if (on(k)) {
                        two_smallest(min0, min1, fabsf(input(k)));
                        neg |= (bits_of(raw[k]) & kSign) >> (31 - k);
                    }
#pragma unroll
                for (int k = 0; k < DM; k++)
                    if (on(k)) {
                        const float a = fabsf(input(k));
                        e0 |= a == min0 ? 1u << k : 0u;
                        e1 |= a == min1 ? 1u << k : 0u;
                    }
                e1 = e0 & (e0 - 1) ? e0 & (e0 - 1) : e1; /* the other holders of an equal minimum */
                e0 &= 0u - e0;
                e1 &= 0u - e1;
            }
            const uint32_t out = __popc(neg) & 1 ? ~neg : neg; /* signs of the outgoing messages */
            const int cl = active ? p.cls[D - (pp ? 0 : 1)] : 0;
            const float beta = sbeta[cl], alpha = salpha[cl];
            const float mu0 = fminf(min0, 127.0f), mu1 = fminf(min1, 127.0f);
            const float pre0 = beta * mu0 - alpha, pre1 = beta * mu1 - alpha;
            const float mag0 = fmaxf(pre0, 0.0f), mag1 = fmaxf(pre1, 0.0f);
            float s0 = 0.0f, s1 = 0.0f; /* gradients of the magnitudes from min0 and from min1 */
            auto pass = [&](int k, float g) { /* g: the gradient of the link's new posterior */
                const bool is = (e0 >> k) & 1u;
                const uint32_t sn = (out << (31 - k)) & kSign;
                const float mag = is ? mag1 : mag0, m = signed_by(mag, sn), post = input(k) + m;
                const float gpost = (post >= -128.0f && post <= 127.0f) ? g : 0.0f;
                const float gmsg = mag <= (sn ? 32.0f : 31.0f) ? go[k] : 0.0f;
                const float gmag = __uint_as_float(bits_of(gpost + gmsg) ^ sn);
                s0 += is ? 0.0f : gmag;
                s1 = is ? gmag : s1;
                go[k] = gpost;
            };
            /* the gradient of the input of link k, once all outputs are in */
            float m0g = 0.0f, m1g = 0.0f;
            auto minimums = [&]() {
                m0g = pre0 > 0.0f && min0 < 127.0f ? s0 * beta * (neg & e0 ? -1.0f : 1.0f) : 0.0f;
                m1g = pre1 > 0.0f && min1 < 127.0f ? s1 * beta * (neg & e1 ? -1.0f : 1.0f) : 0.0f;
            };
            auto gradient = [&](int k) {
                const float g = go[k] + ((e0 >> k) & 1u ? m0g : (e1 >> k) & 1u ? m1g : 0.0f);
                return raw[k] >= -128.0f && raw[k] <= 127.0f ? g : 0.0f;
            };
            if (active) {
                float g[DM];
#pragma unroll
                for (int k = 0; k < DM; k++)
                    if (on(k) && !((early >> k) & 1u))
                        g[k] = at(gP, link_at(c, ent, i, j, k));
#pragma unroll
                for (int k = 0; k < DM; k++)
                    if (on(k) && !((early >> k) & 1u))
                        pass(k, g[k]);
            }
            if (nl > 1) {
                auto levels = [&](auto end) {
                    constexpr int KE = decltype(end)::value < DM ? decltype(end)::value : DM;
                    for (int l = nl - 1; l >= 0; l--) {
                        if (active && lev == l) {
#pragma unroll
                            for (int k = 2; k < KE; k++)
                                if ((early >> k) & 1u)
                                    pass(k, pass_at(tb, first + k - 2, j));
                            minimums();
#pragma unroll
                            for (int k = 2; k < KE; k++)
                                if ((late >> k) & 1u)
                                    pass_at(tb, first + k - 2, j) = gradient(k);
                        }
                        if (l > 0)
                            __syncthreads();
                    }
                };
                const uint32_t any = __reduce_or_sync(0xFFFFFFFFu, late | early);
                if (!(any >> 4))
                    levels(std::integral_constant<int, 4>());
                else if (!(any >> 6))
                    levels(std::integral_constant<int, 6>());
                else
                    levels(std::integral_constant<int, kSharedEnd>());
            } else {
                minimums();
            }
            if (active) {
#pragma unroll
                for (int k = 0; k < DM; k++)
                    if (on(k)) {
                        const float g = gradient(k);
                        if (!((late >> k) & 1u))
                            at(gP, link_at(c, ent, i, j, k)) = g;
                        if (t)
                            __stcs(gMl + kQCl * k, -g);
                    }
                const float w0 = pre0 > 0.0f ? s0 : 0.0f, w1 = pre1 > 0.0f ? s1 : 0.0f;
                const float b = w0 * mu0 + w1 * mu1, a = -(w0 + w1);
                if (pp) {
                    db += b;
                    da += a;
                } else { /* the one check of another degree */
                    atomicAdd(sdb + cl, (double)b);
                    atomicAdd(sda + cl, (double)a);
                }
            }
            /* the sums leave the registers where the layers' degree changes */
            if (i == 0 || (!EXACT && tb.eoff[i] - tb.eoff[i - 1] != D - 2)) {
                for (int o = 16; o > 0; o >>= 1) {
                    db += __shfl_xor_sync(0xFFFFFFFFu, db, o);
                    da += __shfl_xor_sync(0xFFFFFFFFu, da, o);
                }
                if (lane == 0) {
                    atomicAdd(sdb + p.cls[D], db);
                    atomicAdd(sda + p.cls[D], da);
                }
                db = da = 0.0;
            }
            __syncthreads();
        }
        if (j < p.nclass) {
            atomicAdd(p.dbeta + t * p.nclass + j, (float)sdb[j]);
            atomicAdd(p.dalpha + t * p.nclass + j, (float)sda[j]);
        }
        __syncthreads();
    }
}

template <int DM, bool EXACT>
static cudaError_t launch_degree(const LearnedParams& p, bool backward, size_t smem, cudaStream_t s)
{
    if (backward)
        k_learned_bwd<DM, EXACT><<<p.nframes, kLT, smem, s>>>(p);
    else
        k_learned_fwd<DM, EXACT><<<p.nframes, kLT, smem, s>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_learned(const LearnedParams& p, bool backward, const Code& code, cudaStream_t s)
{
    const size_t smem = sizeof(float) * kQCl * kSharedMax + code.ent.size() * sizeof(int32_t) +
                        sizeof(uint16_t) * (code.q + 1) + code.q + code.ent.size() / 2;
    /* the normal DVB-S2 codes' one degree, every other code by its class */
    if (code.cnt_min == code.cnt_max)
        switch (code.deg_max) {
#define DRXG_EXACT(d) \
    case d: return launch_degree<d, true>(p, backward, smem, s);
            DRXG_EXACT(4) DRXG_EXACT(5) DRXG_EXACT(6) DRXG_EXACT(7) DRXG_EXACT(10) DRXG_EXACT(11) DRXG_EXACT(14)
            DRXG_EXACT(18) DRXG_EXACT(22) DRXG_EXACT(27) DRXG_EXACT(30)
#undef DRXG_EXACT
        }
    switch (code.dclass) {
#define DRXG_CLASS(k) \
    case k: return launch_degree<kClassDeg[k], false>(p, backward, smem, s);
        DRXG_CLASS(0) DRXG_CLASS(1) DRXG_CLASS(2) DRXG_CLASS(3) DRXG_CLASS(4) DRXG_CLASS(5)
#undef DRXG_CLASS
    }
    return cudaErrorInvalidValue;
}

}  // namespace drxg
