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
 * the outgoing signs, the link that holds the minimum), exact in fp32.  Degrees
 * are compiled in classes, so a check's links stay in registers.  A layer's
 * checks load every link no earlier check of the layer writes at once; then
 * the wavefront levels in turn load the links that earlier ones wrote.
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

#include "codes.h"
#include "learned.h"

namespace drxg {

constexpr int kLT = 384;
constexpr int kQCl = 360;

__device__ __forceinline__ float clampf(float v, float lo, float hi) { return fminf(fmaxf(v, lo), hi); }
__device__ __forceinline__ float softplus(float u) { return fmaxf(u, 0.0f) + log1pf(expf(-fabsf(u))); }
__device__ __forceinline__ float sigmoid(float u) { return 1.0f / (1.0f + expf(-u)); }

/* The code's link tables, staged in shared memory. */
struct LTables {
    const int2* ent;
    const uint16_t* eoff;
    const uint8_t* nlev;
};

__device__ LTables stage_tables(const DevCode& c, char* smem)
{
    int2* ent = (int2*)smem;
    uint16_t* eoff = (uint16_t*)(ent + c.nent);
    uint8_t* nlev = (uint8_t*)(eoff + c.q + 1);
    for (int k = threadIdx.x; k < c.nent; k += blockDim.x)
        ent[k] = c.ent[k];
    for (int k = threadIdx.x; k <= c.q; k += blockDim.x)
        eoff[k] = c.eoff[k];
    for (int k = threadIdx.x; k < c.q; k += blockDim.x)
        nlev[k] = c.nlev[k];
    return LTables{ ent, eoff, nlev };
}

/* Links of check (i, j): slot 0 = parity, slot 1 = previous parity (absent
 * for (0, 0)), 2.. = information bits (ent: the layer's entries). */
__device__ __forceinline__ int link_var(const DevCode& c, const int2* ent, int i, int j, int slot)
{
    if (slot == 0)
        return c.K + kQCl * i + j;
    if (slot == 1)
        return i ? c.K + kQCl * (i - 1) + j : c.K + kQCl * (c.q - 1) + j - 1;
    const int2 e = ent[slot - 2];
    return e.x + j + (j < e.y ? kQCl : 0);
}

/* The smallest two magnitudes among a check's inputs, the links that hold
 * them (the first of equal ones), those links' signs and all signs' parity. */
struct Node {
    float min0 = 1e30f, min1 = 1e30f;
    int a0 = -1, a1 = -1;
    bool n0 = false, n1 = false, neg = false;
    __device__ __forceinline__ void add(float xv, int k)
    {
        const float a = fabsf(xv);
        const bool n = xv < 0.0f;
        if (a < min0) {
            min1 = min0;
            a1 = a0;
            n1 = n0;
            min0 = a;
            a0 = k;
            n0 = n;
        } else if (a < min1) {
            min1 = a;
            a1 = k;
            n1 = n;
        }
        neg ^= n;
    }
};

/* Loss of the posteriors after an iteration (and a copy of them). */
__device__ float iteration_loss(const DevCode& c, const float* __restrict__ P, const LearnedParams& p, int f,
                                float* __restrict__ copy)
{
    const uint8_t* bits = p.bits + (size_t)f * p.bits_stride;
    float acc = 0.0f;
    for (int v = threadIdx.x; v < c.kldpc; v += blockDim.x) {
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

/* Bound by instruction issue (about 90 a link forward) and, in the layers with
 * wavefront levels, by the warps that wait for a level's few; DRAM 12 %, L2 hits
 * two thirds.  512 normal 2/3 frames, 20 iterations, loss and gradients: 219 ->
 * 73.5 ms.  Before, the backward pass ran every iteration again from a
 * checkpoint of posteriors and messages, and a check's links were arrays
 * indexed at run time, in local memory. */

/* resident CTAs per SM that a degree bound's registers are compiled for */
__host__ __device__ constexpr int fwd_ctas(int dm) { return dm <= 11 ? 3 : dm <= 22 ? 2 : 1; }
__host__ __device__ constexpr int bwd_ctas(int dm) { return dm <= 18 ? 2 : 1; }

template <int DM, bool TRAIN>
__global__ void __launch_bounds__(kLT, fwd_ctas(DM)) k_learned_fwd(LearnedParams p)
{
    extern __shared__ __align__(16) char smem[];
    __shared__ float sbeta[kLearnedMaxClass], salpha[kLearnedMaxClass], red[kLT / 32];
    const DevCode c = *p.code;
    const LTables tb = stage_tables(c, smem);
    const int f = blockIdx.x, j = threadIdx.x;
    const bool active = j < kQCl;
    const size_t E = (size_t)p.DS * c.R;
    float* P = p.P + (size_t)f * c.N;
    uint4* M = p.M + (size_t)f * c.R;
    const __half* src = p.llr + (size_t)f * p.llr_stride;
    for (int v = j; v < c.K; v += blockDim.x)
        P[v] = clampf(__half2float(src[v]), -128.0f, 127.0f);
    for (int k = j; k < c.R; k += blockDim.x)
        P[c.K + kQCl * (k % c.q) + k / c.q] = clampf(__half2float(src[c.K + k]), -128.0f, 127.0f);
    __syncthreads();
    for (int t = 0; t < p.iters; t++) {
        load_params(p, t, sbeta, salpha);
        float* X = TRAIN ? p.Xck + ((size_t)t * p.nframes + f) * E : nullptr;
        uint4 rn = make_uint4(0, 0, 0, 0); /* records and levels one layer ahead */
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
            const int2* ent = tb.ent + tb.eoff[i];
            const int D = tb.eoff[i + 1] - tb.eoff[i] + 2, nl = tb.nlev[i], pos = kQCl * i + j;
            const uint32_t live = ((i | j) ? 0xFFFFFFFFu : ~2u) & (D < 32 ? (1u << D) - 1u : 0xFFFFFFFFu);
            const uint32_t late = (uint32_t)(meta >> 8) & 0xFFFFFFu;
            const int lev = (int)(meta & 0xFF);
            float raw[DM];
            auto load = [&](int k) {
                /* the link's old message */
                const float mag = (int)rec.w == k ? __uint_as_float(rec.y) : __uint_as_float(rec.x);
                const float m = clampf((rec.z >> k) & 1u ? -mag : mag, -32.0f, 31.0f);
                raw[k] = P[link_var(c, ent, i, j, k)] - (t == 0 ? 0.0f : m);
            };
            if (active) {
#pragma unroll
                for (int k = 0; k < DM; k++)
                    if (((live & ~late) >> k) & 1u)
                        load(k);
            }
            for (int l = 0; l < nl; l++) {
                if (active && lev == l) {
                    if (late) {
#pragma unroll
                        for (int k = 2; k < DM; k++)
                            if ((late >> k) & 1u)
                                load(k);
                    }
                    Node n;
#pragma unroll
                    for (int k = 0; k < DM; k++)
                        if ((live >> k) & 1u)
                            n.add(clampf(raw[k], -128.0f, 127.0f), k);
                    const int cl = p.cls[D - ((i | j) ? 0 : 1)];
                    const float beta = sbeta[cl], alpha = salpha[cl];
                    const float mu0 = fminf(n.min0, 127.0f), mu1 = fminf(n.min1, 127.0f);
                    const float mag0 = fmaxf(beta * mu0 - alpha, 0.0f), mag1 = fmaxf(beta * mu1 - alpha, 0.0f);
                    uint32_t signs = 0;
#pragma unroll
                    for (int k = 0; k < DM; k++)
                        if ((live >> k) & 1u) {
                            const float x = clampf(raw[k], -128.0f, 127.0f);
                            const float mag = k == n.a0 ? mag1 : mag0;
                            const bool sneg = n.neg ^ (x < 0.0f);
                            signs |= sneg ? 1u << k : 0u;
                            P[link_var(c, ent, i, j, k)] = clampf(x + (sneg ? -mag : mag), -128.0f, 127.0f);
                            if (TRAIN)
                                __stcs(X + (size_t)k * c.R + pos, raw[k]);
                        }
                    M[pos] = make_uint4(__float_as_uint(mag0), __float_as_uint(mag1), signs, (uint32_t)n.a0);
                }
                __syncthreads();
            }
        }
        float* copy = TRAIN ? p.Pck + ((size_t)t * p.nframes + f) * c.K : nullptr;
        const float l = block_sum(iteration_loss(c, P, p, f, copy), red);
        if (j == 0)
            atomicAdd(p.loss + t, l);
    }
    if (p.post)
        for (int v = j; v < c.kldpc; v += blockDim.x)
            p.post[(size_t)f * c.kldpc + v] = P[v];
}

template <int DM>
__global__ void __launch_bounds__(kLT, bwd_ctas(DM)) k_learned_bwd(LearnedParams p)
{
    extern __shared__ __align__(16) char smem[];
    __shared__ float sbeta[kLearnedMaxClass], salpha[kLearnedMaxClass];
    __shared__ float sdb[kLearnedMaxClass], sda[kLearnedMaxClass];
    const DevCode c = *p.code;
    const LTables tb = stage_tables(c, smem);
    const int f = blockIdx.x, j = threadIdx.x, lane = j & 31;
    const bool active = j < kQCl;
    const size_t E = (size_t)p.DS * c.R;
    float* gP = p.gP + (size_t)f * c.N;
    float* gM = p.gM + (size_t)f * E;
    const uint8_t* bits = p.bits + (size_t)f * p.bits_stride;
    for (int t = p.iters - 1; t >= 0; t--) {
        const bool lastit = t == p.iters - 1;
        if (j < kLearnedMaxClass)
            sdb[j] = sda[j] = 0.0f;
        load_params(p, t, sbeta, salpha);
        /* the gradient of the iteration's loss */
        const float* P = p.Pck + ((size_t)t * p.nframes + f) * c.K;
        const float* X = p.Xck + ((size_t)t * p.nframes + f) * E;
        const float gscale = p.loss_scale * (p.loss_w ? p.loss_w[t] : 1.0f);
        for (int v = j; v < (lastit ? c.N : c.kldpc); v += blockDim.x) {
            float g = 0.0f;
            if (v < c.kldpc) {
                const float sb = ((bits[v >> 3] >> (7 - (v & 7))) & 1) ? -1.0f : 1.0f;
                g = gscale * (-sb * 0.5f) * sigmoid(-sb * __ldcs(P + v) * 0.5f);
            }
            gP[v] = lastit ? g : gP[v] + g;
        }
        __syncthreads();
        float db = 0.0f, da = 0.0f; /* of the layers' class since the last flush */
        for (int i = c.q - 1; i >= 0; i--) {
            const int2* ent = tb.ent + tb.eoff[i];
            const int D = tb.eoff[i + 1] - tb.eoff[i] + 2, nl = tb.nlev[i], pos = kQCl * i + j;
            const uint32_t live = ((i | j) ? 0xFFFFFFFFu : ~2u) & (D < 32 ? (1u << D) - 1u : 0xFFFFFFFFu);
            float raw[DM], go[DM], gmo[DM];
            uint32_t early = 0;
            int lev = 0;
            if (active) {
                const unsigned long long meta = __ldg(c.lmeta + pos);
                early = (uint32_t)(meta >> 32) & 0xFFFFFFu; /* outputs that later checks of the layer read */
                lev = (int)(meta & 0xFF);
#pragma unroll
                for (int k = 0; k < DM; k++)
                    if ((live >> k) & 1u) {
                        raw[k] = __ldcs(X + (size_t)k * c.R + pos);
                        gmo[k] = lastit ? 0.0f : __ldcs(gM + (size_t)k * c.R + pos);
                        if (!((early >> k) & 1u))
                            go[k] = gP[link_var(c, ent, i, j, k)];
                    }
            }
            for (int l = nl - 1; l >= 0; l--) {
                if (active && lev == l) {
                    if (early) {
#pragma unroll
                        for (int k = 2; k < DM; k++)
                            if ((early >> k) & 1u)
                                go[k] = gP[link_var(c, ent, i, j, k)];
                    }
                    Node n;
#pragma unroll
                    for (int k = 0; k < DM; k++)
                        if ((live >> k) & 1u)
                            n.add(clampf(raw[k], -128.0f, 127.0f), k);
                    const int cl = p.cls[D - ((i | j) ? 0 : 1)];
                    const float beta = sbeta[cl], alpha = salpha[cl];
                    const float mu0 = fminf(n.min0, 127.0f), mu1 = fminf(n.min1, 127.0f);
                    const float pre0 = beta * mu0 - alpha, pre1 = beta * mu1 - alpha;
                    const float mag0 = fmaxf(pre0, 0.0f), mag1 = fmaxf(pre1, 0.0f);
                    float s0 = 0.0f, s1 = 0.0f, b = 0.0f, a = 0.0f; /* to the links of the minimums, scale, offset */
#pragma unroll
                    for (int k = 0; k < DM; k++)
                        if ((live >> k) & 1u) {
                            const float x = clampf(raw[k], -128.0f, 127.0f);
                            const bool own = k == n.a0;
                            const bool sneg = n.neg ^ (x < 0.0f);
                            const float mag = own ? mag1 : mag0, m = sneg ? -mag : mag;
                            const float post = x + m;
                            const float gpost = (post >= -128.0f && post <= 127.0f) ? go[k] : 0.0f;
                            const float gmsg = (m >= -32.0f && m <= 31.0f) ? gmo[k] : 0.0f;
                            const float gm = gpost + gmsg, gmag = sneg ? -gm : gm;
                            go[k] = gpost;
                            if ((own ? pre1 : pre0) > 0.0f) {
                                b += gmag * (own ? mu1 : mu0);
                                a -= gmag;
                                if (own)
                                    s1 = gmag;
                                else
                                    s0 += gmag;
                            }
                        }
                    s0 = n.min0 < 127.0f ? s0 * beta * (n.n0 ? -1.0f : 1.0f) : 0.0f;
                    s1 = n.min1 < 127.0f ? s1 * beta * (n.n1 ? -1.0f : 1.0f) : 0.0f;
#pragma unroll
                    for (int k = 0; k < DM; k++)
                        if ((live >> k) & 1u) {
                            const bool inside = raw[k] >= -128.0f && raw[k] <= 127.0f;
                            const float gx = go[k] + (k == n.a0 ? s0 : k == n.a1 ? s1 : 0.0f);
                            const float g = inside ? gx : 0.0f;
                            gP[link_var(c, ent, i, j, k)] = g;
                            if (t)
                                __stcs(gM + (size_t)k * c.R + pos, -g);
                        }
                    if (i | j) {
                        db += b;
                        da += a;
                    } else { /* the one check of another degree */
                        atomicAdd(sdb + cl, b);
                        atomicAdd(sda + cl, a);
                    }
                }
                __syncthreads();
            }
            /* the sums leave the registers where the layers' degree changes */
            if (i == 0 || tb.eoff[i] - tb.eoff[i - 1] != D - 2) {
                for (int o = 16; o > 0; o >>= 1) {
                    db += __shfl_xor_sync(0xFFFFFFFFu, db, o);
                    da += __shfl_xor_sync(0xFFFFFFFFu, da, o);
                }
                if (lane == 0) {
                    atomicAdd(sdb + p.cls[D], db);
                    atomicAdd(sda + p.cls[D], da);
                }
                db = da = 0.0f;
            }
        }
        __syncthreads();
        if (j < p.nclass) {
            atomicAdd(p.dbeta + t * p.nclass + j, sdb[j]);
            atomicAdd(p.dalpha + t * p.nclass + j, sda[j]);
        }
        __syncthreads();
    }
}

template <int DM>
static cudaError_t launch_degree(const LearnedParams& p, bool backward, size_t smem, cudaStream_t s)
{
    if (backward)
        k_learned_bwd<DM><<<p.nframes, kLT, smem, s>>>(p);
    else if (p.Xck)
        k_learned_fwd<DM, true><<<p.nframes, kLT, smem, s>>>(p);
    else
        k_learned_fwd<DM, false><<<p.nframes, kLT, smem, s>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_learned(const LearnedParams& p, bool backward, int dclass, int nent, int q, cudaStream_t s)
{
    const size_t smem = sizeof(int2) * (size_t)nent + sizeof(uint16_t) * (q + 1) + q;
    static_assert(kNumClasses == 6 && kClassDeg[5] == 32, "degree classes");
    switch (dclass) {
    case 0: return launch_degree<kClassDeg[0]>(p, backward, smem, s);
    case 1: return launch_degree<kClassDeg[1]>(p, backward, smem, s);
    case 2: return launch_degree<kClassDeg[2]>(p, backward, smem, s);
    case 3: return launch_degree<kClassDeg[3]>(p, backward, smem, s);
    case 4: return launch_degree<kClassDeg[4]>(p, backward, smem, s);
    case 5: return launch_degree<kClassDeg[5]>(p, backward, smem, s);
    }
    return cudaErrorInvalidValue;
}

}  // namespace drxg
