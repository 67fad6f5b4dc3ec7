/*
 * BCH decoding of DVB-S2 BBFRAMEs on the GPU (EN 302 307-1 5.3.1), with the
 * reference's results (libdvbrx/src/bch.c:189-290, declared
 * libdvbrx/include/dvbrx/fec.h:27-37): the corrected codeword in place and
 * the number of corrected bits, or -1 with the word untouched.
 *
 * The code: g(x) = product of the minimal polynomials of alpha^(2i+1),
 * i < t, over GF(2^16) (normal frames, primitive x^16+x^5+x^3+x^2+1) or
 * GF(2^14) (short frames, x^14+x^5+x^3+x+1); W = deg g = 16 t or 14 t parity
 * bits; codewords of nbch = kldpc bits, MSB first, the highest degree first.
 *
 * k_bch_remainder: the remainders c(x) x^W mod g(x) of a batch, 16 or 32 lanes
 * per frame; a zero remainder ends the frame (no error), the others are
 * queued.  The same kernel over the message bytes encodes.
 * k_bch_correct: up to four queued frames per CTA: syndromes and
 * Berlekamp-Massey by a warp each, then the roots of one locator after the
 * other over the whole field; when those at positions of the shortened code
 * number the degree, their bits are flipped.  For a correctable word the locator
 * is unique, so the result does not depend on how it was found.
 */
#include <cuda_pipeline.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <string>
#include <vector>

#include "../../include/dvbrx_b200.h"
#include "handle.h"

namespace drxg {

constexpr int kBchMaxT = 12;
constexpr int kBchWords = 3;     /* 64-bit words of the largest remainder register (192 bits) */
constexpr int kRemMaxWarps = 16; /* warps per CTA of the remainder kernel */
constexpr int kFixThreads = 128; /* threads per CTA of the correction kernel */

/* Lanes that share one frame in the remainder kernel, and the steps of the
 * pairwise combination of their partial remainders. */
constexpr int kWideLanes = 32, kWideLevels = 5;
constexpr int kThinLanes = 16, kThinLevels = 4;

struct BchDev {
    int m, q, t, W, nbch;
    int nwide, nthin;              /* 32-bit words per lane with 32 and with 16 lanes per frame */
    const unsigned long long* step; /* [256][NW]: the entries of the division step */
    const unsigned long long* comb; /* [9][16 NW][16][NW]: the nibble tables of the combinations, 5 wide, 4 thin */
    const uint16_t* log;           /* q + 1 */
    const uint32_t* syn;  /* [64 NW][8]: for every remainder bit its part of S_1, S_3 .., two in a word */
    const uint16_t* anf;  /* [12][697 or 470]: x^k's coefficients at the subsets of 1, 2 and 3 bits */
    const uint32_t* sets; /* the bits i | j << 8 | k << 16 of every subset */
};

struct BchBatch {
    BchDev c;
    uint8_t* cw;
    size_t stride;
    int32_t* result;
    int nframes;
    unsigned long long* rem; /* per frame: its remainder, where it is not zero */
    int32_t* queue;          /* frames with a remainder */
    int* count;              /* queue length, zeroed before the remainder kernel */
};

/*
 * Remainders.  The frames' bytes are cut into LPF chunks of n 32-bit words
 * (zeros in front of the first byte), one lane per chunk; a lane divides its
 * chunk by g(x) a word per step,
 *     r <- (r << 32) ^ T(top word of r ^ word),
 * T the XOR of one entry from each of six tables (6, 6, 5, 5, 5 and 5 bits of
 * the word).  Every entry is kept 16 times, replica k in the 8-byte bank pair
 * k, so the 16 lanes of a half warp read their entries without bank
 * conflicts.  Then the lanes of a frame combine their remainders in pairs,
 * left x^(32 n 2^s) + right, the product a sum of nibble-table entries that
 * the lanes of the pair share out.
 * Bound by shared-memory reads: 18 reads of 256 bytes per step and warp, 36
 * of the 44 cycles that the load unit needs with the row loads; one thread per
 * frame over byte tables, as it was, waited for each step's reads in turn on
 * 64 threads' tables per CTA.  A decode call of 4096 normal 3/5 words without
 * errors 0.260 -> 0.061 ms, 0.042 of it this kernel; parity of 999 normal 9/10
 * words 0.532 -> 0.016 ms.  Half warps (n =
 * 76 words) against whole warps (40) at 2048 words: 31 against 27 us, at 4096
 * no difference, so half a warp is taken once the batch has no warp for each.
 */
constexpr int kChunks = 6;
__host__ __device__ constexpr int chunk_bits(int c) { return c < 2 ? 6 : 5; }
__host__ __device__ constexpr int chunk_shift(int c) { return c < 2 ? 26 - 6 * c : 15 - 5 * (c - 2); }
__host__ __device__ constexpr int chunk_first(int c) { return c < 2 ? 64 * c : 128 + 32 * (c - 2); } /* entry */
constexpr int kEntries = 256; /* entries of the six tables */

/* bytes of an entry's 16 replicas (a power of two, so that an index is placed by a shift) */
template <int NW>
constexpr int kEntryBytes = NW == 3 ? 512 : 256;
template <int NW>
constexpr size_t rem_smem(int levels)
{
    return (size_t)kEntries * kEntryBytes<NW> + (size_t)levels * NW * 16 * 16 * NW * 8;
}

/* the 16 bytes at p (16-byte aligned), those outside [lo, hi) as zeros */
__device__ __forceinline__ uint4 block_at(const uint8_t* p, const uint8_t* lo, const uint8_t* hi)
{
    if (p >= lo && p + 16 <= hi)
        return __ldg((const uint4*)p);
    uint32_t w[4] = { 0, 0, 0, 0 };
    if (p < hi && p + 16 > lo) {
#pragma unroll
        for (int k = 0; k < 16; k++)
            if (p + k >= lo && p + k < hi)
                w[k / 4] |= (uint32_t)p[k] << (8 * (k % 4));
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

__device__ __forceinline__ unsigned long long lds64(uint32_t a)
{
    unsigned long long v;
    asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"(a));
    return v;
}

template <int NW, int LPF, bool ENCODE>
__global__ void __launch_bounds__(32 * kRemMaxWarps) k_bch_remainder(BchBatch b, int nbytes)
{
    constexpr int LEVELS = LPF == kWideLanes ? kWideLevels : kThinLevels;
    constexpr int FPW = 32 / LPF;        /* frames per warp */
    constexpr int NIB = 16 * NW;         /* nibbles of a remainder */
    constexpr int EB = kEntryBytes<NW>;
    extern __shared__ __align__(16) char smem[];
    unsigned long long* comb = (unsigned long long*)(smem + (size_t)kEntries * EB); /* [LEVELS][NIB][16][NW] */
    const BchDev& c = b.c;
    const int t = threadIdx.x;

    /* the combination tables arrive while the frames are divided */
    const char* src = (const char*)(c.comb + (LPF == kWideLanes ? 0 : (size_t)kWideLevels * NIB * 16 * NW));
    for (int k = t; k < LEVELS * NIB * NW; k += blockDim.x) /* 128 bytes each */
#pragma unroll
        for (int i = 0; i < 8; i++)
            __pipeline_memcpy_async((char*)comb + 16 * (k + i * LEVELS * NIB * NW),
                                    src + 16 * (k + i * LEVELS * NIB * NW), 16);
    __pipeline_commit();
#pragma unroll 12
    for (int k = t; k < kEntries * NW * 16; k += blockDim.x) {
        const int r = k & 15, ew = k >> 4;
        *(unsigned long long*)(smem + (size_t)(ew / NW) * EB + (ew % NW) * 128 + 8 * r) = __ldg(c.step + ew);
    }
    __syncthreads();

    const int lane = t & 31, sub = lane % LPF, nwarps = blockDim.x >> 5;
    const int n = LPF == kWideLanes ? c.nwide : c.nthin;
    const uint32_t tab = (uint32_t)__cvta_generic_to_shared(smem) + 8u * (lane & 15);
    /* the frames of a round go around the CTAs first, then around their warps */
    const int per_round = gridDim.x * nwarps * FPW;
    for (int round = 0; round * per_round < b.nframes; round++) {
        const int f0 = round * per_round + ((t >> 5) * gridDim.x + blockIdx.x) * FPW;
        const int f = f0 + lane / LPF;
        /* lanes past the batch take an empty row */
        uint8_t* row = b.cw + (size_t)min(f, b.nframes - 1) * b.stride;
        const uint8_t *lo = row, *hi = f < b.nframes ? row + nbytes : row;
        const ptrdiff_t s = (ptrdiff_t)4 * n * sub - ((ptrdiff_t)4 * n * LPF - nbytes);
        const uint8_t* a = row + s;
        const int ws = (int)((uintptr_t)a & 15) >> 2, by = (int)((uintptr_t)a & 3);
        /* big-endian word from bytes by .. by + 3 of a word pair */
        const uint32_t swap = 0x0123u + 0x1111u * (uint32_t)by;
        const uint8_t* p = a - ((uintptr_t)a & 15);
        /* blocks in flight: four steps take less than a load's latency */
        uint4 cur = block_at(p, lo, hi), nxt = block_at(p + 16, lo, hi), far[2];
#pragma unroll
        for (int k = 0; k < 2; k++)
            far[k] = block_at(p + 32 + 16 * k, lo, hi);
        unsigned long long r[NW];
#pragma unroll
        for (int w = 0; w < NW; w++)
            r[w] = 0;
        for (int i = 0; i < n && f0 < b.nframes; i += 4) {
            const uint32_t q[8] = { cur.x, cur.y, cur.z, cur.w, nxt.x, nxt.y, nxt.z, nxt.w };
            uint32_t u[6], x[5];
#pragma unroll
            for (int k = 0; k < 6; k++)
                u[k] = (ws & 2) ? q[k + 2] : q[k];
#pragma unroll
            for (int k = 0; k < 5; k++)
                x[k] = (ws & 1) ? u[k + 1] : u[k];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const uint32_t top = (uint32_t)(r[0] >> 32) ^ __byte_perm(x[k], x[k + 1], swap);
                unsigned long long d[NW];
#pragma unroll
                for (int w = 0; w < NW; w++)
                    d[w] = r[w] << 32 | (w + 1 < NW ? r[w + 1 < NW ? w + 1 : w] >> 32 : 0ull);
#pragma unroll
                for (int ch = 0; ch < kChunks; ch++) {
                    constexpr int LB = EB == 512 ? 9 : 8;
                    const int sh = chunk_shift(ch);
                    const uint32_t m = ((1u << chunk_bits(ch)) - 1u) << LB;
                    const uint32_t at = ((sh >= LB ? top >> (sh >= LB ? sh - LB : 0) : top << (sh >= LB ? 0 : LB - sh)) & m) + tab;
#pragma unroll
                    for (int w = 0; w < NW; w++)
                        d[w] ^= lds64(at + (uint32_t)(chunk_first(ch) * EB + 128 * w));
                }
#pragma unroll
                for (int w = 0; w < NW; w++)
                    r[w] = d[w];
            }
            cur = nxt;
            nxt = far[0];
            far[0] = far[1];
            p += 16;
            far[1] = i + 12 < n ? block_at(p + 48, lo, hi) : make_uint4(0, 0, 0, 0);
        }
        if (round == 0) {
            __pipeline_wait_prior(0);
            __syncthreads();
        }
        if (f0 >= b.nframes)
            continue;
        /* pairs of chunks, then pairs of pairs: left x^(32 n 2^s) + right; each of the
         * G lanes of a group takes PER nibbles of the left remainder */
#pragma unroll
        for (int s2 = 0; s2 < LEVELS; s2++) {
            constexpr unsigned ALL = 0xFFFFFFFFu;
            const int G = 2 << s2, gi = sub & (G - 1), PER = (NIB + G - 1) / G;
            const bool right = (sub >> s2) & 1;
            unsigned long long L[NW], acc[NW];
#pragma unroll
            for (int w = 0; w < NW; w++) {
                const unsigned long long o = __shfl_xor_sync(ALL, r[w], 1 << s2);
                L[w] = right ? o : r[w];
                acc[w] = gi == 0 ? o : 0ull; /* the group's first lane is a left one: o is the right sum */
            }
            /* this lane's nibbles, at the low end of m (at most 96 bits) */
            const int bit = 4 * PER * gi, wd = bit >> 6;
            unsigned long long lo = L[NW - 1], hi = NW > 1 ? L[NW - 2] : 0ull;
#pragma unroll
            for (int w = 1; w < NW; w++) {
                lo = wd == w ? L[NW - 1 - w] : lo;
                hi = wd == w ? (w + 1 < NW ? L[NW - 2 - w < 0 ? 0 : NW - 2 - w] : 0ull) : hi;
            }
            const int sh = bit & 63;
            const unsigned long long m0 = sh ? lo >> sh | hi << (64 - sh) : lo, m1 = hi >> sh;
            const uint32_t m[3] = { (uint32_t)m0, (uint32_t)(m0 >> 32), (uint32_t)m1 };
            const uint32_t tb = (uint32_t)__cvta_generic_to_shared(comb) + (uint32_t)(s2 * NIB + PER * gi) * 16 * NW * 8;
            if (NIB % G == 0 || PER * gi < NIB) {
#pragma unroll
                for (int k = 0; k < PER; k++) {
                    const uint32_t e = tb + ((m[k / 8] >> (4 * (k % 8))) & 15u) * (NW * 8u);
#pragma unroll
                    for (int w = 0; w < NW; w++)
                        acc[w] ^= lds64(e + (uint32_t)(16 * NW * 8 * k + 8 * w));
                }
            }
#pragma unroll
            for (int o = 1; o < G; o <<= 1)
#pragma unroll
                for (int w = 0; w < NW; w++)
                    acc[w] ^= __shfl_xor_sync(ALL, acc[w], o);
#pragma unroll
            for (int w = 0; w < NW; w++)
                r[w] = acc[w];
        }
        if (f >= b.nframes)
            continue;
        if (ENCODE) {
            for (int k = sub; k < c.W / 8; k += LPF) {
                unsigned long long word = r[0];
#pragma unroll
                for (int w = 1; w < NW; w++)
                    word = k / 8 == w ? r[w] : word;
                row[nbytes + k] = (uint8_t)(word >> (56 - 8 * (k % 8)));
            }
        } else if (sub == 0) {
            unsigned long long any = 0;
#pragma unroll
            for (int w = 0; w < NW; w++)
                any |= r[w];
            b.result[f] = any ? -1 : 0; /* the correction kernel changes it where it corrects */
            if (any) {
#pragma unroll
                for (int w = 0; w < NW; w++)
                    b.rem[(size_t)f * NW + w] = r[w];
                const int at = atomicAdd(b.count, 1);
                if (at < b.nframes) /* always, unless another call on the handle overlaps */
                    b.queue[at] = f;
            }
        }
    }
}

/*
 * Correction of the frames with a remainder R != 0, a CTA taking up to four:
 * each warp finds one frame's locator, from the syndromes S_j = R(alpha^j)
 * alpha^(-jW) (odd j; even ones by squaring) by Berlekamp-Massey with lane k
 * holding coefficient k (a serial chain of table lookups), then all warps find
 * the roots of one locator after the other.
 *
 * Roots.  A polynomial of degree at most 12 is, in the bits of its argument,
 * of degree at most 3 (an exponent's degree is its number of ones, and 7 and
 * 11 have three).  So the locator's value at every x is the sum over the
 * subsets of x's bits of at most three elements of 16-bit coefficients (697
 * for GF(2^16), 470 for GF(2^14)), themselves sums of the locator's
 * coefficients times constants of the field.  Each thread fixes seven high bits of x, sums the
 * coefficients over them, and walks the other 2^9 (2^7) points by halving:
 * fixing a bit adds the coefficients that hold it to those that do not, and
 * sixteen words remain, each with the two values of bit 0.  About two
 * instructions per point take the place of twelve table lookups at every
 * position of the code.
 * Bound by latency: up to four CTAs an SM, the locator 6 us and the roots 5 us
 * of dependent steps; a lone frame 26 us, 1024 frames with errors 50 us.  The
 * evaluation at every position with one thread's Berlekamp-Massey before it
 * took 1.1 ms for the 1024 (normal 3/5), 3.3 ms for 4096 frames with 12 errors.
 */
__host__ __device__ constexpr int pair_at(int i, int j) { return j * (j - 1) / 2 + i; } /* i < j */
__host__ __device__ constexpr int triple_at(int i, int j, int k) { return k * (k - 1) * (k - 2) / 6 + pair_at(i, j); }

constexpr int kMaxPts = 16 + 120 + 560;

/* Carry-less product of two 16-bit values, by masked integer products (the
 * constant-time method of Pornin's BearSSL, "ctmul").  The factors are taken
 * apart into bits four apart, so that the at most four terms of a result bit add
 * up without a carry into the next bit of its class: about 30 independent
 * instructions, where a product through logarithms waits for two loads from a
 * table too large for L1. */
__device__ __forceinline__ uint32_t clmul(uint32_t a, uint32_t b)
{
    const uint32_t a0 = a & 0x1111u, a1 = a & 0x2222u, a2 = a & 0x4444u, a3 = a & 0x8888u;
    const uint32_t b0 = b & 0x1111u, b1 = b & 0x2222u, b2 = b & 0x4444u, b3 = b & 0x8888u;
    return (((a0 * b0) ^ (a1 * b3) ^ (a2 * b2) ^ (a3 * b1)) & 0x11111111u) |
           (((a0 * b1) ^ (a1 * b0) ^ (a2 * b3) ^ (a3 * b2)) & 0x22222222u) |
           (((a0 * b2) ^ (a1 * b1) ^ (a2 * b0) ^ (a3 * b3)) & 0x44444444u) |
           (((a0 * b3) ^ (a1 * b2) ^ (a2 * b1) ^ (a3 * b0)) & 0x88888888u);
}

/* A product, or a sum of products, as an element of GF(2^16) (x^16 = x^5 +
 * x^3 + x^2 + 1) or GF(2^14) (x^14 = x^5 + x^3 + x + 1). */
template <int M>
__device__ __forceinline__ uint32_t gred(uint32_t z)
{
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const uint32_t h = z >> M;
        z = (z & ((1u << M) - 1u)) ^ h ^ h << (M == 16 ? 2 : 1) ^ h << 3 ^ h << 5;
    }
    return z;
}

template <int M>
__device__ __forceinline__ uint32_t gmul(uint32_t a, uint32_t b)
{
    return gred<M>(clmul(a, b));
}

constexpr int kFixWarps = kFixThreads / 32;

struct FixShared {
    uint32_t L[kFixWarps][kBchMaxT + 2]; /* the locators' coefficients, up to a common factor */
    int frame[kFixWarps], len[kFixWarps];
    uint16_t a[kMaxPts];                        /* coefficients of the subsets of 1, 2 and 3 bits */
    uint32_t p0, p1[15], p2[105], p3[455];      /* coefficients over bits 1 .., (bit 0 = 0) | (bit 0 = 1) << 16 */
    int nroots, roots[kBchMaxT + 1], npos, pos[kBchMaxT + 1];
};

/* The zeros among sixteen words; out of line, so that the walk stays in the
 * instruction cache (inlined sixteen times, it doubled the kernel's time). */
__device__ __noinline__ void note_zeros(const uint32_t* u, FixShared& s, int x)
{
    for (int w = 0; w < 16; w++) {
        if (!(u[w] & 0xFFFFu))
            s.roots[min(atomicAdd(&s.nroots, 1), kBchMaxT)] = x + 2 * w;
        if (!(u[w] >> 16))
            s.roots[min(atomicAdd(&s.nroots, 1), kBchMaxT)] = x + 2 * w + 1;
    }
}

/* The zeros of a cubic with coefficients c0, c1, c2 and s.p3 among the 2^D
 * words from point x on (two points a word). */
template <int D>
__device__ __forceinline__ void walk_cubic(uint32_t c0, const uint32_t* c1, const uint32_t* c2, FixShared& s, int x)
{
    if constexpr (D == 4) {
        uint32_t v[16];
#pragma unroll
        for (int w = 0; w < 16; w++)
            v[w] = 0;
        v[0] = c0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            v[1 << i] = c1[i];
#pragma unroll
            for (int j = i + 1; j < 4; j++) {
                v[1 << i | 1 << j] = c2[pair_at(i, j)];
#pragma unroll
                for (int k = j + 1; k < 4; k++)
                    v[1 << i | 1 << j | 1 << k] = s.p3[triple_at(i, j, k)];
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int w = 0; w < 16; w++)
                if ((w >> i) & 1)
                    v[w] ^= v[w ^ (1 << i)];
        uint32_t m = v[0];
#pragma unroll
        for (int w = 1; w < 16; w++)
            m = __vminu2(m, v[w]);
        if (!(m & 0xFFFFu) || !(m >> 16)) { /* at most 12 times in all */
            uint32_t u[16];
#pragma unroll
            for (int w = 0; w < 16; w++)
                u[w] = v[w];
            note_zeros(u, s, x);
        }
    } else {
        /* the top bit clear, then set */
        walk_cubic<D - 1>(c0, c1, c2, s, x);
        uint32_t d1[D - 1], d2[(D - 1) * (D - 2) / 2];
#pragma unroll
        for (int i = 0; i < D - 1; i++) {
            d1[i] = c1[i] ^ c2[pair_at(i, D - 1)];
#pragma unroll
            for (int j = i + 1; j < D - 1; j++)
                d2[pair_at(i, j)] = c2[pair_at(i, j)] ^ s.p3[triple_at(i, j, D - 1)];
        }
        walk_cubic<D - 1>(c0 ^ c1[D - 1], d1, d2, s, x + (1 << D));
    }
}

template <int M>
__global__ void __launch_bounds__(kFixThreads, 4) k_bch_correct(BchBatch b)
{
    constexpr int H = 7;         /* bits of x fixed by the thread */
    constexpr int D = M - 1 - H; /* bits walked, besides bit 0 */
    static_assert(1 << H == kFixThreads, "one thread per value of the high bits");
    __shared__ FixShared s;
    const BchDev& c = b.c;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int n = min(b.count[0], b.nframes);
    const int nw = c.W > 128 ? 3 : 2;
    uint32_t mk[H];
#pragma unroll
    for (int h = 0; h < H; h++)
        mk[h] = 0u - (((uint32_t)t >> h) & 1u);
    for (int q0 = blockIdx.x; q0 < n; q0 += kFixWarps * gridDim.x) {
        /* each warp finds one frame's locator */
        const int qi = q0 + warp * gridDim.x;
        int f = qi < n ? b.queue[qi] : -1;
        f = f < b.nframes ? f : -1; /* a row of another batch, if calls on the handle overlap */
        if (lane == 0)
            s.frame[warp] = f;
        if (f >= 0) {
            /* S_1, S_3 ..: two in a word */
            uint32_t so[6] = { 0, 0, 0, 0, 0, 0 };
#pragma unroll
            for (int w = 0; w < kBchWords; w++) {
                if (w >= nw)
                    break;
                const unsigned long long word = b.rem[(size_t)f * nw + nw - 1 - w]; /* the low one first */
#pragma unroll
                for (int h = 0; h < 2; h++)
                    if ((word >> (32 * h + lane)) & 1) {
                        const uint4* r = (const uint4*)(c.syn + 8 * (64 * w + 32 * h + lane));
                        const uint4 x = __ldg(r), y = __ldg(r + 1);
                        so[0] ^= x.x;
                        so[1] ^= x.y;
                        so[2] ^= x.z;
                        so[3] ^= x.w;
                        so[4] ^= y.x;
                        so[5] ^= y.y;
                    }
            }
            /* lane j holds S_j: the odd ones from the sums, S_2j = S_j^2 */
            uint32_t S = 0;
#pragma unroll
            for (int k = 0; k < 6; k++) {
                const uint32_t v = __reduce_xor_sync(0xFFFFFFFFu, so[k]);
                S = lane == 4 * k + 1 ? v & 0xFFFFu : lane == 4 * k + 3 ? v >> 16 : S;
            }
#pragma unroll
            for (int k = 1; k <= 4; k++) {
                const uint32_t v = __shfl_sync(0xFFFFFFFFu, S, lane >> 1);
                S = __ffs(lane) == k + 1 ? gmul<M>(v, v) : S;
            }
            if (lane > 2 * c.t)
                S = 0;
            /* Berlekamp-Massey without divisions: the shortest LFSR L(x), up to a
             * factor, that generates S_1 .. S_2t.  With S_2j = S_j^2 every second
             * discrepancy is zero.  The running length can pass t + 1 on uncorrectable
             * words: updates stop at degree t + 1, as in bch.c (the word has failed then) */
            uint32_t L = lane == 0, B = L;
            uint32_t bd = 1; /* the discrepancy that B belongs to */
            int len = 0, shift = 1;
            for (int k = 0; k < 2 * c.t; k += 2) {
                const uint32_t sk = __shfl_sync(0xFFFFFFFFu, S, (k + 1 - lane) & 31); /* lane 0: S_(k+1) */
                const uint32_t d = __reduce_xor_sync(0xFFFFFFFFu, lane <= len ? gmul<M>(L, sk) : 0u);
                if (!d) {
                    shift += 2;
                    continue;
                }
                const uint32_t bs = __shfl_sync(0xFFFFFFFFu, B, (lane - shift) & 31);
                const uint32_t old = L;
                L = gred<M>(clmul(L, bd) ^ (lane >= shift && lane <= c.t + 1 ? clmul(bs, d) : 0u));
                if (2 * len <= k) {
                    len = k + 1 - len;
                    B = old;
                    bd = d;
                    shift = 2;
                } else {
                    shift += 2;
                }
            }
            if (lane <= kBchMaxT + 1)
                s.L[warp][lane] = L;
            if (lane == 0)
                s.len[warp] = len;
        }
        __syncthreads();
        /* the CTA finds the roots of one locator after the other */
#pragma unroll 1
        for (int g4 = 0; g4 < kFixWarps; g4++) {
            const int f = s.frame[g4], len = s.len[g4];
            if (f < 0 || len > c.t) /* no frame, or not correctable: the result stays -1 */
                continue;
            const uint32_t* L = s.L[g4]; /* zero above len */
            if (t == 0)
                s.nroots = s.npos = 0;
            /* the locator's coefficients: those of its powers that have subsets of the size */
            constexpr int F2 = M, F3 = M + M * (M - 1) / 2, NP = F3 + M * (M - 1) * (M - 2) / 6;
            auto term = [&](int power, int k) { return clmul(__ldg(c.anf + (power - 1) * NP + k), L[power]); };
#pragma unroll 3
            for (int k = F3 + t; k < NP; k += kFixThreads)
                s.a[k] = (uint16_t)gred<M>(term(7, k) ^ term(11, k));
            for (int k = t; k < F3; k += kFixThreads) {
                uint32_t v = term(3, k) ^ term(5, k) ^ term(6, k) ^ term(7, k) ^ term(9, k) ^ term(10, k) ^
                             term(11, k) ^ term(12, k);
                if (k < F2)
                    v ^= term(1, k) ^ term(2, k) ^ term(4, k) ^ term(8, k);
                s.a[k] = (uint16_t)gred<M>(v);
            }
            __syncthreads();
            /* for both values of bit 0: the subsets without it */
#pragma unroll
            for (int k = t; k < NP; k += kFixThreads) {
                const uint32_t ix = __ldg(c.sets + k);
                const int i = ix & 255, j = (ix >> 8) & 255, l = ix >> 16;
                const uint32_t v = s.a[k];
                if (i == 0)
                    continue;
                if (k < F2)
                    s.p1[i - 1] = v | (v ^ s.a[F2 + pair_at(0, i)]) << 16;
                else if (k < F3)
                    s.p2[pair_at(i - 1, j - 1)] = v | (v ^ s.a[F3 + triple_at(0, i, j)]) << 16;
                else
                    s.p3[triple_at(i - 1, j - 1, l - 1)] = v * 0x00010001u;
            }
            if (t == 0)
                s.p0 = L[0] | (L[0] ^ s.a[0]) << 16;
            __syncthreads();
            /* this thread's coefficients: summed over the subsets of its high bits */
            uint32_t c0 = s.p0, c1[D], c2[D * (D - 1) / 2];
#pragma unroll
            for (int g = 0; g < H; g++) {
                c0 ^= mk[g] & s.p1[D + g];
#pragma unroll
                for (int h = g + 1; h < H; h++) {
                    const uint32_t gh = mk[g] & mk[h];
                    c0 ^= gh & s.p2[pair_at(D + g, D + h)];
#pragma unroll
                    for (int u = h + 1; u < H; u++)
                        c0 ^= gh & mk[u] & s.p3[triple_at(D + g, D + h, D + u)];
                }
            }
#pragma unroll
            for (int i = 0; i < D; i++) {
                c1[i] = s.p1[i];
#pragma unroll
                for (int g = 0; g < H; g++) {
                    c1[i] ^= mk[g] & s.p2[pair_at(i, D + g)];
#pragma unroll
                    for (int h = g + 1; h < H; h++)
                        c1[i] ^= mk[g] & mk[h] & s.p3[triple_at(i, D + g, D + h)];
                }
#pragma unroll
                for (int j = i + 1; j < D; j++) {
                    uint32_t v = s.p2[pair_at(i, j)];
#pragma unroll
                    for (int g = 0; g < H; g++)
                        v ^= mk[g] & s.p3[triple_at(i, j, D + g)];
                    c2[pair_at(i, j)] = v;
                }
            }
            walk_cubic<D>(c0, c1, c2, s, t << (D + 1));
            __syncthreads();
            if (t < min(s.nroots, kBchMaxT)) { /* the root alpha^-p is the error at position p */
                const int lx = (int)__ldg(c.log + s.roots[t]);
                const int p = lx ? c.q - lx : 0;
                if (p < c.nbch)
                    s.pos[atomicAdd(&s.npos, 1)] = p;
            }
            __syncthreads();
            if (t == 0 && s.npos == len) { /* distinct positions: one thread flips them */
                uint8_t* w = b.cw + (size_t)f * b.stride;
                for (int k = 0; k < len; k++) {
                    const int bit = c.nbch - 1 - s.pos[k];
                    w[bit / 8] ^= (uint8_t)(0x80u >> (bit % 8));
                }
                b.result[f] = len;
            }
            __syncthreads();
        }
        __syncthreads();
    }
}

}  // namespace drxg

using namespace drxg;

struct drx_bch {
    int device = 0;
    int sms = 0;
    int short_frame = 0, m = 0, q = 0, t = 0, kbch = 0, nbch = 0, W = 0;
    void* blob = nullptr;
    BchDev dev{};
    cudaStream_t stream = nullptr;
    unsigned long long* rem = nullptr;
    int32_t* queue = nullptr;
    int* count = nullptr;
    size_t cap = 0;
    uint8_t* d_cw = nullptr;
    int32_t* d_res = nullptr;
};

namespace {

/* Field and division tables.  A register of NW words is left-aligned (x^(W-1)
 * at its top bit).  tab: the 256 entries of the division step (sums of x^(W + i)
 * mod g for the bits i of a message word), then for every level s of the two
 * combinations (32 lanes per frame, 16 lanes) and every nibble of the register,
 * the low one first, the images of its 16 values times x^(32 n 2^s) mod g. */
bool bch_tables(drx_bch* b, std::vector<unsigned long long>& tab, std::vector<uint16_t>& ex, std::vector<uint16_t>& lg,
                std::vector<uint32_t>& sets, std::vector<uint16_t>& anf, std::vector<uint32_t>& syn)
{
    const int m = b->m, q = b->q;
    const unsigned prim = b->short_frame ? 0x402Bu : 0x1002Du;
    ex.assign(2 * (size_t)q, 0);
    lg.assign((size_t)q + 1, 0);
    unsigned x = 1;
    for (int i = 0; i < q; i++) {
        ex[i] = ex[i + q] = (uint16_t)x;
        lg[x] = (uint16_t)i;
        x <<= 1;
        if (x >> m)
            x ^= prim;
    }
    auto mul = [&](uint16_t a, uint16_t c) -> uint16_t { return a && c ? ex[lg[a] + lg[c]] : 0; };
    /* g(x): product of the minimal polynomials of alpha^i, i = 1, 3, .., 2t-1 */
    std::vector<uint8_t> g(1, 1);
    for (int i = 1; i < 2 * b->t; i += 2) {
        std::vector<uint16_t> p(1, 1);
        int e = i % q;
        do {
            const uint16_t beta = ex[e];
            p.push_back(0);
            for (size_t k = p.size() - 1; k > 0; k--)
                p[k] = p[k - 1] ^ mul(p[k], beta);
            p[0] = mul(p[0], beta);
            e = (2 * e) % q;
        } while (e != i % q);
        std::vector<uint8_t> r(g.size() + p.size() - 1, 0);
        for (size_t a = 0; a < g.size(); a++)
            if (g[a])
                for (size_t c = 0; c < p.size(); c++)
                    r[a + c] ^= (uint8_t)(p[c] & 1);
        g = r;
    }
    b->W = (int)g.size() - 1;
    if (b->W > 64 * kBchWords || b->W != b->nbch - b->kbch)
        return false;
    const int W = b->W, NW = W > 128 ? 3 : 2, pad = 64 * NW - W;
    auto words_of = [&](int lanes) { return ((b->nbch / 8 + 4 * lanes - 1) / (4 * lanes) + 3) & ~3; };
    b->dev.nwide = words_of(kWideLanes);
    b->dev.nthin = words_of(kThinLanes);
    /* powers of x mod g up to the highest image */
    unsigned long long low[kBchWords] = { 0, 0, 0 }, r[kBchWords] = { 0, 0, 0 };
    for (int k = 0; k < W; k++)
        if (g[k])
            low[NW - 1 - (k + pad) / 64] |= 1ull << ((k + pad) % 64);
    r[NW - 1 - pad / 64] = 1ull << (pad % 64); /* x^0 */
    constexpr int kLevels = kWideLevels + kThinLevels;
    std::vector<unsigned long long> rows((size_t)(32 + kLevels * 64 * NW) * NW, 0);
    int first[kLevels], last = W + 32;
    for (int s = 0; s < kLevels; s++) {
        first[s] = s < kWideLevels ? 32 * b->dev.nwide << s : 32 * b->dev.nthin << (s - kWideLevels);
        last = std::max(last, first[s] + W);
    }
    std::vector<uint8_t> used((size_t)last, 0); /* the powers that are images */
    memset(&used[W], 1, 32);
    for (int s = 0; s < kLevels; s++)
        memset(&used[first[s]], 1, W);
    for (int e = 0; e < last; e++) {
        auto put = [&](size_t row) {
            for (int w = 0; w < NW; w++)
                rows[row * NW + w] = r[w];
        };
        if (e >= W && e < W + 32)
            put(e - W);
        for (int s = 0; used[e] && s < kLevels; s++)
            if (e >= first[s] && e < first[s] + W)
                put(32 + (size_t)s * 64 * NW + pad + (e - first[s]));
        const bool top = r[0] >> 63;
        for (int w = 0; w < NW; w++)
            r[w] = (r[w] << 1 | (w + 1 < NW ? r[w + 1] >> 63 : 0)) ^ (top ? low[w] : 0ull);
    }
    /* entry v of a table over `bits` register bits from row r0 on: the sum of v's rows */
    auto sum = [&](unsigned long long* out, size_t r0, int bits, int v) {
        for (int i = 0; i < bits; i++)
            if ((v >> i) & 1)
                for (int w = 0; w < NW; w++)
                    out[w] ^= rows[(r0 + i) * NW + w];
    };
    tab.assign((size_t)(kEntries + kLevels * 16 * NW * 16) * NW, 0);
    for (int c = 0; c < kChunks; c++)
        for (int v = 0; v < 1 << chunk_bits(c); v++)
            sum(&tab[(size_t)(chunk_first(c) + v) * NW], chunk_shift(c), chunk_bits(c), v);
    for (int k = 0; k < kLevels * 16 * NW; k++)
        for (int v = 0; v < 16; v++)
            sum(&tab[((size_t)kEntries + 16 * (size_t)k + v) * NW], 32 + 4 * (size_t)k, 4, v);
    /* what every register bit adds to S_j = R(alpha^j) alpha^(-jW) */
    syn.assign((size_t)64 * NW * 8, 0);
    for (int i = 0; i < W; i++)
        for (int k = 0; k < b->t; k++) {
            const int e = ((2 * k + 1) * (i - W) % q + q) % q;
            syn[(size_t)(i + pad) * 8 + k / 2] |= (uint32_t)ex[e] << (16 * (k % 2));
        }
    /* the subsets of one, two and three bits, and the coefficients of x^1 .. x^12
     * at them: sums of the values at their subsets (x^k is 0 at 0) */
    sets.clear();
    for (int i = 0; i < m; i++)
        sets.push_back((unsigned)i);
    for (int j = 0; j < m; j++)
        for (int i = 0; i < j; i++)
            sets.push_back((unsigned)(i | j << 8));
    for (int k = 0; k < m; k++)
        for (int j = 0; j < k; j++)
            for (int i = 0; i < j; i++)
                sets.push_back((unsigned)(i | j << 8 | k << 16));
    const int n1 = m, n2 = n1 + m * (m - 1) / 2, n3 = (int)sets.size();
    anf.assign((size_t)12 * n3, 0);
    std::vector<unsigned> lx(n3); /* logarithm of the element with the subset's bits */
    for (int n = 0; n < n3; n++)
        lx[n] = lg[1u << (sets[n] & 255) | (n < n1 ? 0u : 1u << (sets[n] >> 8 & 255)) | (n < n2 ? 0u : 1u << (sets[n] >> 16))];
    std::vector<uint16_t> v(n3); /* x^k there */
    for (int k = 1; k <= 12; k++) {
        uint16_t* a = &anf[(size_t)(k - 1) * n3];
        for (int n = 0; n < n3; n++)
            v[n] = ex[(size_t)lx[n] * k % q];
        for (int n = 0; n < n3; n++) {
            const int i = sets[n] & 255, j = sets[n] >> 8 & 255, l = sets[n] >> 16;
            a[n] = v[n];
            if (n >= n1)
                a[n] ^= v[i] ^ v[j];
            if (n >= n2)
                a[n] ^= v[l] ^ v[n1 + pair_at(i, j)] ^ v[n1 + pair_at(i, l)] ^ v[n1 + pair_at(j, l)];
        }
    }
    return true;
}

bool bch_scratch(drx_bch* b, size_t n)
{
    if (b->cap >= n)
        return true;
    cudaStreamSynchronize(b->stream);
    cudaFree(b->rem);
    cudaFree(b->queue);
    b->rem = nullptr;
    b->queue = nullptr;
    b->cap = 0;
    if (!cuda_check(drxg::dev_malloc(&b->rem, n * kBchWords * sizeof(unsigned long long)), "cudaMalloc(bch)") ||
        !cuda_check(drxg::dev_malloc(&b->queue, n * sizeof(int32_t)), "cudaMalloc(bch)"))
        return false;
    b->cap = n;
    return true;
}

template <int NW, int LPF, bool ENCODE>
cudaError_t launch_remainder(const BchBatch& p, int nbytes, int sms, cudaStream_t s)
{
    constexpr int fpw = 32 / LPF;
    const size_t smem = rem_smem<NW>(LPF == kWideLanes ? kWideLevels : kThinLevels);
    cudaError_t e = cudaFuncSetAttribute(k_bch_remainder<NW, LPF, ENCODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess)
        return e;
    const int grid = std::min((p.nframes + fpw - 1) / fpw, sms);
    k_bch_remainder<NW, LPF, ENCODE><<<grid, 32 * kRemMaxWarps, smem, s>>>(p, nbytes);
    return cudaGetLastError();
}

template <bool ENCODE>
cudaError_t remainders(const drx_bch* b, const BchBatch& p, int nbytes, cudaStream_t s)
{
    /* A warp per frame while every frame has a warp at once, half a warp per
     * frame beyond */
    const bool thin = p.nframes > kRemMaxWarps * b->sms;
    if (b->W > 128)
        return thin ? launch_remainder<3, kThinLanes, ENCODE>(p, nbytes, b->sms, s)
                    : launch_remainder<3, kWideLanes, ENCODE>(p, nbytes, b->sms, s);
    return thin ? launch_remainder<2, kThinLanes, ENCODE>(p, nbytes, b->sms, s)
                : launch_remainder<2, kWideLanes, ENCODE>(p, nbytes, b->sms, s);
}

int bch_enqueue(drx_bch* b, uint8_t* cw, size_t stride, int32_t* result, int nframes, cudaStream_t s)
{
    if (nframes <= 0)
        return 0;
    if (!cw || !result || stride < (size_t)(b->nbch / 8)) {
        set_error("drx_bch_decode_device: bad arguments");
        return -1;
    }
    if (!bch_scratch(b, (size_t)nframes))
        return -1;
    BchBatch p{};
    p.c = b->dev;
    p.cw = cw;
    p.stride = stride;
    p.result = result;
    p.nframes = nframes;
    p.rem = b->rem;
    p.queue = b->queue;
    p.count = b->count;
    /* in every call: a length left by one that failed or overlapped another ends with it */
    if (!cuda_check(cudaMemsetAsync(b->count, 0, sizeof(int), s), "cudaMemsetAsync") ||
        !cuda_check(remainders<false>(b, p, b->nbch / 8, s), "BCH remainder"))
        return -1;
    const int grid = std::min(nframes, 4 * b->sms);
    if (b->m == 16)
        k_bch_correct<16><<<grid, kFixThreads, 0, s>>>(p);
    else
        k_bch_correct<14><<<grid, kFixThreads, 0, s>>>(p);
    return cuda_check(cudaGetLastError(), "BCH correction") ? 0 : -1;
}

}  // namespace

extern "C" {

drx_bch* drx_bch_new(const drx_fec_params* p)
{
    if (!p || p->t < 1 || p->t > kBchMaxT || p->kldpc <= p->kbch || p->kldpc % 8) {
        set_error("drx_bch_new: not a DVB-S2 BCH code");
        return nullptr;
    }
    drx_bch* b = new drx_bch();
    b->short_frame = p->short_frame ? 1 : 0;
    b->m = b->short_frame ? 14 : 16;
    b->q = (1 << b->m) - 1;
    b->t = p->t;
    b->kbch = p->kbch;
    b->nbch = p->kldpc;
    std::vector<unsigned long long> tab;
    std::vector<uint16_t> ex, lg;
    std::vector<uint32_t> sets, syn;
    std::vector<uint16_t> anf;
    if (!bch_tables(b, tab, ex, lg, sets, anf, syn)) {
        set_error("drx_bch_new: parity length does not match the code");
        delete b;
        return nullptr;
    }
    bool ok = cuda_check(cudaGetDevice(&b->device), "cudaGetDevice") &&
              cuda_check(cudaDeviceGetAttribute(&b->sms, cudaDevAttrMultiProcessorCount, b->device), "attribute") &&
              cuda_check(cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking), "cudaStreamCreate");
    const size_t o_syn = tab.size() * 8, o_sets = o_syn + syn.size() * 4, o_anf = o_sets + sets.size() * 4,
                 o_lg = o_anf + anf.size() * 2, total = o_lg + lg.size() * 2 + 64;
    ok = ok && cuda_check(drxg::dev_malloc(&b->blob, total), "cudaMalloc(bch tables)") &&
         cuda_check(drxg::dev_malloc(&b->count, sizeof(int)), "cudaMalloc") &&
         cuda_check(drxg::dev_malloc(&b->d_cw, (size_t)b->nbch / 8), "cudaMalloc") &&
         cuda_check(drxg::dev_malloc(&b->d_res, sizeof(int32_t)), "cudaMalloc");
    if (ok) {
        char* base = (char*)b->blob;
        std::vector<char> host(total);
        memcpy(host.data(), tab.data(), tab.size() * 8);
        memcpy(host.data() + o_syn, syn.data(), syn.size() * 4);
        memcpy(host.data() + o_sets, sets.data(), sets.size() * 4);
        memcpy(host.data() + o_anf, anf.data(), anf.size() * 2);
        memcpy(host.data() + o_lg, lg.data(), lg.size() * 2);
        ok = cuda_check(cudaMemcpy(base, host.data(), total, cudaMemcpyHostToDevice), "cudaMemcpy");
        b->dev.m = b->m;
        b->dev.q = b->q;
        b->dev.t = b->t;
        b->dev.W = b->W;
        b->dev.nbch = b->nbch;
        b->dev.step = (const unsigned long long*)base;
        b->dev.comb = b->dev.step + (size_t)kEntries * (b->W > 128 ? 3 : 2);
        b->dev.syn = (const uint32_t*)(base + o_syn);
        b->dev.sets = (const uint32_t*)(base + o_sets);
        b->dev.anf = (const uint16_t*)(base + o_anf);
        b->dev.log = (const uint16_t*)(base + o_lg);
    }
    if (!ok) {
        drx_bch_free(b);
        return nullptr;
    }
    return b;
}

void drx_bch_free(drx_bch* b)
{
    if (!b)
        return;
    if (b->stream)
        cudaStreamSynchronize(b->stream);
    cudaFree(b->blob);
    cudaFree(b->rem);
    cudaFree(b->queue);
    cudaFree(b->count);
    cudaFree(b->d_cw);
    cudaFree(b->d_res);
    if (b->stream)
        cudaStreamDestroy(b->stream);
    delete b;
}

int drx_bch_decode_device(drx_bch* b, uint8_t* cw, size_t stride, int32_t* result, int nframes, void* stream)
{
    if (!b) {
        set_error("drx_bch_decode_device: NULL handle");
        return -1;
    }
    return bch_enqueue(b, cw, stride, result, nframes, stream ? (cudaStream_t)stream : b->stream);
}

int drx_bch_encode_device(drx_bch* b, uint8_t* cw, size_t stride, int nframes, void* stream)
{
    if (!b || (nframes > 0 && !cw) || stride < (size_t)(b->nbch / 8) || b->kbch % 8) {
        set_error("drx_bch_encode_device: bad arguments");
        return -1;
    }
    if (nframes <= 0)
        return 0;
    BchBatch p{};
    p.c = b->dev;
    p.cw = cw;
    p.stride = stride;
    p.nframes = nframes;
    return cuda_check(remainders<true>(b, p, b->kbch / 8, stream ? (cudaStream_t)stream : b->stream), "BCH encode")
               ? 0
               : -1;
}

int drx_bch_test_left_over(drx_bch* b, int frames)
{
    if (!b || frames < 0) {
        set_error("drx_bch_test_left_over: NULL handle or a negative count");
        return -1;
    }
    return cuda_check(cudaMemcpy(b->count, &frames, sizeof(int), cudaMemcpyHostToDevice), "cudaMemcpy") ? 0 : -1;
}

int drx_bch_decode(drx_bch* b, uint8_t* cw)
{
    if (!b || !cw) {
        set_error("drx_bch_decode: NULL argument");
        return -1;
    }
    const size_t nb = (size_t)b->nbch / 8;
    int32_t res = -1;
    if (!cuda_check(cudaMemcpyAsync(b->d_cw, cw, nb, cudaMemcpyHostToDevice, b->stream), "cudaMemcpyAsync") ||
        bch_enqueue(b, b->d_cw, nb, b->d_res, 1, b->stream) ||
        !cuda_check(cudaMemcpyAsync(&res, b->d_res, sizeof(int32_t), cudaMemcpyDeviceToHost, b->stream),
                    "cudaMemcpyAsync") ||
        !cuda_check(cudaStreamSynchronize(b->stream), "BCH decode"))
        return -1;
    if (res > 0 &&
        !cuda_check(cudaMemcpy(cw, b->d_cw, nb, cudaMemcpyDeviceToHost), "cudaMemcpy"))
        return -1;
    return res;
}

}  // extern "C"
