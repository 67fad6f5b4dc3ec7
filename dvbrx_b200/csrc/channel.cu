/*
 * Synthetic DVB-S2 frames on the GPU: the input source of the benchmark and
 * of the learned decoder's training.  One CTA per frame:
 *
 *   1. information bits from a counter-based generator (Philox4x32-10,
 *      Salmon et al., "Parallel random numbers: as easy as 1, 2, 3", SC 2011)
 *      keyed by (seed, frame);
 *   2. the systematic encoder of EN 302 307-1 5.3.2 in the layer form of the
 *      decoder's code, on 32 bits at a time: the checks (i, 0 .. 359) of layer i
 *      sum rotations of the layer's 360-bit groups; the accumulator over
 *      k = q*j + i is a prefix sum over the layers of every column j, then over
 *      the columns' sums;
 *   3. the bit interleaver and mapping of the MODCOD (bit b of symbol j is
 *      codeword bit order[b] * nsym + j; QPSK: bits 2j, 2j+1), unit average
 *      energy points;
 *   4. complex AWGN of power n0 = 10^(-Es/N0 / 10) per symbol (Box-Muller);
 *   5. the max-log demapper with the reference receiver's scale and
 *      quantiser (libdvbrx/src/demap.c:32-34,225-229,491-533): LLR =
 *      quantise(2/n0 * (min_{bit=1} d - min_{bit=0} d)), d = |p|^2 - 2 Re(y p*)
 *      formed as x*(-2 re) + (y*(-2 im) + |p|^2) with fused multiply-adds,
 *      QPSK in closed form 2/n0 * 4/sqrt(2) * component; quantise = clamp to
 *      +-127 then round half to even.  Optionally the unquantised values as
 *      FP16 (for training).
 */
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "channel.h"

namespace drxg {

constexpr int kChThreads = 512;
constexpr int kChWarps = kChThreads / 32;
constexpr int kQCc = 360;
constexpr int kColWords = 12;  /* 32-bit words of a layer's 360 columns */
constexpr int kRowWords = 13;  /* their stride: consecutive layers in different banks */

/* Philox4x32-10 */
struct P4 {
    uint32_t x, y, z, w;
};
__device__ __forceinline__ P4 philox(P4 c, uint32_t k0, uint32_t k1)
{
#pragma unroll
    for (int r = 0; r < 10; r++) {
        const uint32_t hi0 = __umulhi(0xD2511F53u, c.x), lo0 = 0xD2511F53u * c.x;
        const uint32_t hi1 = __umulhi(0xCD9E8D57u, c.z), lo1 = 0xCD9E8D57u * c.z;
        c = P4{ hi1 ^ c.y ^ k0, lo1, hi0 ^ c.w ^ k1, lo0 };
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
    return c;
}

__device__ __forceinline__ float u01(uint32_t v) { return ((float)(v >> 8) + 0.5f) * (1.0f / 16777216.0f); }

__device__ __forceinline__ int quantise(float v)
{
    v = fminf(fmaxf(v, -127.0f), 127.0f);
    return __float2int_rn(v);
}

/* Smallest distances over the points whose label bit b is 0 and 1 (the order
 * of a minimum does not matter): every point for up to 32, from 64 on groups
 * of 16 with the low four bits inside a group and the others from the groups'
 * minima. */
template <int BITS>
__device__ __forceinline__ void distances(const ChannelParams& p, float x, float y, float* m0, float* m1)
{
#pragma unroll
    for (int b = 0; b < BITS; b++)
        m0[b] = m1[b] = 3.0e38f;
    constexpr int GB = BITS < 5 ? BITS : BITS < 6 ? 5 : 4; /* label bits inside a group */
#pragma unroll 1
    for (int g = 0; g < (1 << (BITS - GB)); g++) {
        float all = 3.0e38f;
#pragma unroll
        for (int q = 0; q < (1 << GB); q++) {
            const int pt = (g << GB) | q;
            const float d = fmaf(x, p.ar[pt], fmaf(y, p.ai[pt], p.e[pt]));
            if (GB < BITS)
                all = fminf(all, d);
#pragma unroll
            for (int L = 0; L < GB; L++) {
                if ((q >> L) & 1)
                    m1[BITS - 1 - L] = fminf(m1[BITS - 1 - L], d);
                else
                    m0[BITS - 1 - L] = fminf(m0[BITS - 1 - L], d);
            }
        }
#pragma unroll
        for (int L = GB; L < BITS; L++) {
            const bool one = (g >> (L - GB)) & 1;
            m1[BITS - 1 - L] = one ? fminf(m1[BITS - 1 - L], all) : m1[BITS - 1 - L];
            m0[BITS - 1 - L] = one ? m0[BITS - 1 - L] : fminf(m0[BITS - 1 - L], all);
        }
    }
}

/* Bound by the symbols' arithmetic (about 200 instructions each: Philox, the
 * noise's logarithm and sine, the distances); the encoder on words is a few
 * per cent of it.  1024 normal 2/3 8PSK frames 1.158 -> 0.231 ms: one byte per
 * codeword bit (65 KB a frame, three CTAs an SM, a byte gathered per link) and
 * minimums indexed at run time, in local memory, before. */
template <int BITS>
__global__ void __launch_bounds__(kChThreads) k_channel(const __grid_constant__ ChannelParams p)
{
    extern __shared__ __align__(16) uint32_t words[]; /* information bits, then [q][kRowWords] parity */
    __shared__ uint32_t column[kColWords];
    __shared__ float2 point[1 << BITS];
    const DevCode c = *p.code;
    const int f = blockIdx.x / p.parts, part = blockIdx.x - f * p.parts;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const uint32_t k0 = (uint32_t)p.seed, k1 = (uint32_t)(p.seed >> 32);
    const int blocks = (c.K + 127) / 128;
    uint32_t* info = words;
    uint32_t* par = words + 4 * blocks + 4;

    /* 1. information bits: counter (frame, block of 128 bits, stream 0) */
    for (int b = t; b < blocks; b += kChThreads) {
        const P4 r = philox(P4{ (uint32_t)b, (uint32_t)f, 0u, 0x494E464Fu }, k0, k1);
        info[4 * b] = r.x;
        info[4 * b + 1] = r.y;
        info[4 * b + 2] = r.z;
        info[4 * b + 3] = r.w;
    }
    for (int k = t; k < (1 << BITS); k += kChThreads)
        point[k] = make_float2(-0.5f * p.ar[k], -0.5f * p.ai[k]);
    __syncthreads();

    /* 2. layer i's checks 32 w .. 32 w + 31: the bits (j - a) mod 360 of its groups */
    auto bits_at = [&](int pos) { /* 32 information bits from bit pos on */
        return __funnelshift_r(info[pos >> 5], info[(pos >> 5) + 1], pos & 31);
    };
    for (int k = t; k < c.q * kColWords; k += kChThreads) {
        const int i = k / kColWords, w = k - i * kColWords;
        uint32_t v = 0;
        const int e1 = c.eoff[i + 1];
        for (int e = c.eoff[i]; e < e1; e++) {
            const int2 en = __ldg(c.ent + e); /* (360 g - a, a) */
            const int base = en.x + en.y;
            int s = 32 * w - en.y;
            s += s < 0 ? kQCc : 0;
            uint32_t x = bits_at(base + s);
            if (s > kQCc - 32) { /* the group's first bits follow its last */
                const int n = kQCc - s;
                x = (x & ((1u << n) - 1u)) | bits_at(base) << n;
            }
            v ^= x;
        }
        par[i * kRowWords + w] = w == kColWords - 1 ? v & 0xFFu : v;
    }
    __syncthreads();
    /* prefix sums over the layers: a warp per word, every lane a run of layers */
    for (int w = warp; w < kColWords; w += kChWarps) {
        const int run = (c.q + 31) / 32, lo = min(c.q, lane * run), hi = min(c.q, lo + run);
        uint32_t sum = 0;
        for (int i = lo; i < hi; i++)
            sum ^= par[i * kRowWords + w];
        uint32_t before = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, before, o);
            before ^= lane >= o ? u : 0u;
        }
        if (lane == 31)
            column[w] = before; /* the columns' sums */
        before ^= sum;
        for (int i = lo; i < hi; i++) {
            before ^= par[i * kRowWords + w];
            par[i * kRowWords + w] = before;
        }
    }
    __syncthreads();
    if (warp == 0) { /* the columns before each column */
        const uint32_t own = lane < kColWords ? column[lane] : 0u;
        uint32_t v = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
            v ^= v << o;
        const uint32_t odd = __ballot_sync(0xFFFFFFFFu, v >> 31); /* words with an odd sum */
        if (__popc(odd & ((1u << lane) - 1u)) & 1)
            v = ~v;
        if (lane < kColWords)
            column[lane] = v ^ own;
    }
    __syncthreads();

    /* information bits out, packed MSB first */
    if (p.info && part == 0) {
        uint8_t* dst = p.info + (size_t)f * p.info_stride;
        for (int B = t; B < c.nbytes; B += kChThreads) {
            uint32_t v = __brev(info[B >> 2] >> (8 * (B & 3))) >> 24;
            if (8 * B + 8 > c.kldpc)
                v &= 0xFF00u >> (c.kldpc - 8 * B);
            dst[B] = (uint8_t)v;
        }
    }

    /* codeword bit: information bit, or the parity of column k / q, layer k % q */
    const uint32_t qm = 0xFFFFFFFFu / (uint32_t)c.q + 1u;
    auto bit = [&](int pos) -> uint32_t {
        if (pos < c.K)
            return (info[pos >> 5] >> (pos & 31)) & 1u;
        const uint32_t k = (uint32_t)(pos - c.K), j = __umulhi(k, qm), i = k - j * c.q;
        return ((par[i * kRowWords + (j >> 5)] ^ column[j >> 5]) >> (j & 31)) & 1u;
    };

    /* 3-5. symbols, noise, demapper */
    const float n0 = p.n0, sig = sqrtf(0.5f * n0), kk = 2.0f / n0;
    int8_t* llr = p.llr ? p.llr + (size_t)f * p.llr_stride : nullptr;
    __half* llrh = p.llr_f16 ? p.llr_f16 + (size_t)f * p.llr_f16_stride : nullptr;
    const int nsym = (c.N + BITS - 1) / BITS;
    for (int j = part * kChThreads + t; j < nsym; j += p.parts * kChThreads) {
        const P4 r = philox(P4{ (uint32_t)j, (uint32_t)f, 1u, 0x5eedu }, k0, k1);
        const float rad = sqrtf(-2.0f * logf(u01(r.x)));
        float sn, cs;
        sincospif(2.0f * u01(r.y), &sn, &cs);
        const float nx = sig * rad * cs, ny = sig * rad * sn;
        if (BITS == 2) {
            const uint32_t b0 = bit(2 * j), b1 = bit(2 * j + 1);
            const float re = point[0].x, im = point[0].y;
            const float x = (b0 ? -re : re) + nx;
            const float y = (b1 ? -im : im) + ny;
            const float kq = kk * 4.0f * 0.70710678118654752f;
            const float vx = __fmul_rn(kq, x), vy = __fmul_rn(kq, y);
            if (llr) {
                llr[2 * j] = (int8_t)quantise(vx);
                llr[2 * j + 1] = (int8_t)quantise(vy);
            }
            if (llrh) {
                llrh[2 * j] = __float2half_rn(vx);
                llrh[2 * j + 1] = __float2half_rn(vy);
            }
        } else {
            int label = 0;
#pragma unroll
            for (int b = 0; b < BITS; b++) {
                const int pos = p.order[b] * nsym + j;
                label = (label << 1) | (pos < c.N ? (int)bit(pos) : 0);
            }
            const float2 pt = point[label];
            const float x = pt.x + nx, y = pt.y + ny;
            float m0[BITS], m1[BITS];
            distances<BITS>(p, x, y, m0, m1);
#pragma unroll
            for (int b = 0; b < BITS; b++) {
                const int pos = p.order[b] * nsym + j;
                if (pos >= c.N)
                    continue;
                const float v = __fmul_rn(kk, __fsub_rn(m1[b], m0[b]));
                if (llr)
                    llr[pos] = (int8_t)quantise(v);
                if (llrh)
                    llrh[pos] = __float2half_rn(v);
            }
        }
    }
}

cudaError_t launch_channel(const ChannelParams& p0, int nframes, int N, int K, int q, int sms, cudaStream_t s)
{
    ChannelParams p = p0;
    const size_t smem = 4 * ((size_t)4 * ((K + 127) / 128) + 4 + (size_t)kRowWords * q);
    /* CTAs per frame: a few frames alone would leave SMs idle, and encoding a frame
     * again takes less time than the symbols handed over; one once the frames fill
     * the four CTAs of every SM */
    const int most = ((N + p.bits - 1) / p.bits + kChThreads - 1) / kChThreads;
    p.parts = std::max(1, std::min(std::min(most, 16), 4 * sms / nframes));
    const int grid = nframes * p.parts;
    switch (p.qpsk ? 2 : p.bits) {
    case 2:
        k_channel<2><<<grid, kChThreads, smem, s>>>(p);
        break;
    case 3:
        k_channel<3><<<grid, kChThreads, smem, s>>>(p);
        break;
    case 4:
        k_channel<4><<<grid, kChThreads, smem, s>>>(p);
        break;
    case 5:
        k_channel<5><<<grid, kChThreads, smem, s>>>(p);
        break;
    case 6:
        k_channel<6><<<grid, kChThreads, smem, s>>>(p);
        break;
    case 7:
        k_channel<7><<<grid, kChThreads, smem, s>>>(p);
        break;
    case 8:
        k_channel<8><<<grid, kChThreads, smem, s>>>(p);
        break;
    default:
        return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace drxg
