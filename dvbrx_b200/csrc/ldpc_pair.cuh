/*
 * Plain decoder, frame-pair variant (device code, included by the
 * ldpc_pair_k*.cu files, which instantiate the kernels in parts so that
 * they compile in parallel; ldpc_pair.cu holds the host side): the same arithmetic as ldpc_decode.cu
 * (bit-exact to libdvbrx/src/ldpc.c), two frames per CTA.
 *
 * SIMD within a register: each 32-bit register carries the same quantity for
 * two frames as two halves, lane A in the low one and lane B in the high one,
 * every value of the decoder being exact in one (PairCheck).  One instruction
 * stream decodes two frames.
 *
 * Shared memory holds both frames' posteriors interleaved: the 16-bit word
 * v holds the posterior of variable v, plus 128, for lane A (low byte) and
 * lane B (high byte): K information bits, then R parity bits in layer order.
 *
 * A check node runs on one thread: 360 of the 384 threads hold the 360
 * checks of a layer, every link of a check in registers, no shuffles (two
 * threads per check, combining their minimums with a shuffle round, ran
 * 17-22 % slower on 3/5 and 18/30: twice the per-check set-up and finish
 * work for the same link work).  Levelled layers run in phases (layer_pair): the
 * wavefront levels carry only the links two checks of the layer share.  The
 * thread of a check stores its compressed messages for both frames in one
 * 8-byte record: per lane min0 (6 bits) | min1 << 6 | index << 12, then the
 * sign bits.
 *
 * Frames stream through the two lanes independently: when a lane's frame
 * passes the syndrome check or reaches max_iter, its results are written
 * and the lane takes the next frame of the batch (its first iteration reads
 * zero messages), so a converged frame never waits for its neighbour.
 * Every DVB-S2, S2X and T2 code runs here (check degrees up to 30; message
 * records of 16 bytes above degree 16).
 */
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "codes.h"
#include "ldpc_device.h"

namespace drxg {

constexpr int kQCp = 360;
/* a kernel compiled for LS reads late and writes early only link slots
 * 2 .. 2 LS + 1 */
constexpr int kLateSlotsMax = 6;

/* PRMT in its default mode: a selector nibble with bit 3 set replicates the
 * sign bit of the selected byte.  (__byte_perm keeps only the low 3 bits of
 * each nibble, so the sign-replicating forms need the instruction itself.) */
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel)
{
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}
/* 0xFFFF in each lane whose bit 15 is set */
__device__ __forceinline__ uint32_t lmask(uint32_t v) { return prmt(v, 0, 0xBB99); }
/* 16-bit shared-memory accesses at a 32-bit shared address, to and from whole
 * registers (a 16-bit register would cost a conversion on either side) */
__device__ __forceinline__ uint32_t lds16(uint32_t a)
{
    uint32_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts16(uint32_t a, uint32_t v)
{
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "r"(v));
}

/*
 * One check node (i, j) for both lanes, on one thread: link slots
 * k = 0 .. S-1.  Slot 0 is the parity bit, slot 1 the previous parity bit
 * (absent for (0, 0)), 2 + e information entry e of the layer.  DM is the
 * node degree.  The node state lives in registers across the phases of its layer
 * (see layer_pair).  Slot masks and the message index keep slot k at bit k.
 *
 * The full passes run every slot without branches: a slot that is not a link,
 * or whose bit another check of the layer shares (taken in after the layer's
 * levels), enters the minimums above every real magnitude; stores are
 * predicated.
 *
 * Sign bits of a record: the 16 slots of a word in the byte layout
 * byte 0 = lane A even slots, byte 1 = lane A odd slots, byte 2 = lane B
 * even slots, byte 3 = lane B odd slots, slot 2s (2s + 1) at bit 7 - s of
 * its byte: one PRMT takes the signs of two slots of both lanes there, and one
 * shift brings a slot's back to the halves' sign bits.
 */
/* A check's message record: 8 bytes up to degree 16 (per lane min0, min1
 * and a 4-bit index in one word, 16 sign bits per lane in the other); 16
 * bytes above (min0 and min1; sign bits of slots 0-15 and of slots 16-31;
 * the index, 16 bits per lane). */
template <bool WIDE>
using PairRec = typename std::conditional<WIDE, uint4, uint2>::type;

/* The learned magnitudes of the current iteration (learned kernels): byte
 * 1024 h + 128 k + m = min(learned_mag(m, word of lane h's row and degree
 * class k), 255) for capped minimums m = 0..127.  A magnitude of 255 or more
 * saturates every posterior it meets and is capped at 32 in the record, so
 * the cap at 255 changes no result.  Rebuilt at the start of each learned
 * iteration (iterate_pair). */
static __shared__ uint8_t s_learn_lut[2 * kLearnClasses * 128];

/* the learned magnitudes of capped minimums c (both lanes, 0..127) from the
 * check's class table at index t of s_learn_lut (lane A; lane B at t + 1024) */
__device__ __forceinline__ uint32_t learned_lut(uint32_t c, uint32_t t)
{
    return (uint32_t)s_learn_lut[t + (c & 0xFFFFu)] | (uint32_t)s_learn_lut[t + 1024u + (c >> 16)] << 16;
}

/*
 * Values are halves in units of 1/256, exact: a posterior P is kept as the byte
 * u = P + 128, which one PRMT makes the half 4 + u/256, and
 *     x = sat((4 + u/256) - (4 + m)) - 1/2 = (P - m)/256,
 * the saturating add being the clamp at -128 and one minimum
 * the clamp at 127 (255/256 before the half is taken off).  |x| is an operand
 * modifier of the minimum, a link's message magnitude is a fused multiply-add
 * of the comparison's 1.0, min0 + f (min1 - min0), its sign one LOP3.  The
 * record's index is a slot that holds min0 (a tie makes min1 = min0, and then
 * which one changes no message), collected by a fused multiply-add per slot in
 * chains of about seven.
 *
 * Bound by issue: the decoder on 16-bit integers had 39 instructions of the
 * integer pipe per link and frame pair of normal 3/5 (counted over a launch, level
 * steps and syndrome included; the pipe 72 % busy, the FMA pipe 13 %), this form
 * 25, its adds and selects on the FMA pipe (63 and 47 %).  us of the GPU per
 * frame-iteration before and after this step alone: S2X 18/30 0.305 and 0.206, normal 2/3 0.297
 * and 0.279, 8/9 0.264 and 0.223, 9/10 0.331 and 0.257, short 1/2 0.086 and
 * 0.072, 3/5 0.143 and 0.117; normal 3/5 8PSK, 4096 frames over its waterfall
 * 37.4 and 31.3 ms.  Measured and not kept: link addresses two in a register or
 * formed again where 80 registers spill (short 5/6 and 8/9, normal 4/5; fewer
 * spills, 8 to 25 % slower), one CTA per SM for those.
 */
__device__ __forceinline__ __half2 h2(uint32_t a) { return *(const __half2*)&a; }
__device__ __forceinline__ uint32_t u2(__half2 a) { return *(const uint32_t*)&a; }
constexpr uint32_t kH127 = 0x37F037F0u;    /* 127/256 */
constexpr uint32_t kHHalf = 0x38003800u;   /* 1/2 */
constexpr uint32_t kH31 = 0x2FC02FC0u;     /* 31/256 */
constexpr uint32_t kH32 = 0x30003000u;     /* 32/256 */
constexpr uint32_t kHFour = 0x44004400u;   /* 4: its low byte counts in 1/256 */
constexpr uint32_t kH255 = 0x3BF83BF8u;    /* 255/256 */
constexpr uint32_t kHNegFour = 0xC400C400u;
constexpr uint32_t kHOne = 0x3C003C00u;    /* above every magnitude */
constexpr uint32_t kHSign = 0x80008000u;
constexpr uint32_t kHNegUnit = 0x9C009C00u; /* -1/256 */

__device__ __forceinline__ uint32_t h_add(uint32_t a, uint32_t b) { return u2(__hadd2(h2(a), h2(b))); }
/* bytes in both lanes as halves in 1/256, and back */
__device__ __forceinline__ uint32_t h_of_int(uint32_t v) { return h_add(v | kHFour, kHNegFour); }
__device__ __forceinline__ uint32_t h_to_int(uint32_t v) { return h_add(v, kHFour) & 0x00FF00FFu; }
/* x from a posterior word (two bytes u), whose halves' upper bytes come from
 * four (0x44 in its byte 1), and minus 4 minus the message */
__device__ __forceinline__ uint32_t h_input(uint32_t raw, uint32_t four, uint32_t cm)
{
    const __half2 z = __hadd2_sat(h2(prmt(raw, four, 0x5150)), h2(cm));
    return u2(__hsub2(__hmin2(z, h2(kH255)), h2(kHHalf)));
}
/* the new posterior's two bytes from x and the message */
__device__ __forceinline__ uint32_t h_output(uint32_t x, uint32_t m)
{
    const __half2 z = __hmin2(__hadd2_sat(h2(x), h2(h_add(m, kHHalf))), h2(kH255));
    return prmt(h_add(u2(z), kHFour), 0, 0x0020);
}
__device__ __forceinline__ uint32_t h_abs(uint32_t x) { return u2(__habs2(h2(x))); }
__device__ __forceinline__ uint32_t h_min(uint32_t a, uint32_t b) { return u2(__hmin2(h2(a), h2(b))); }
__device__ __forceinline__ uint32_t h_max(uint32_t a, uint32_t b) { return u2(__hmax2(h2(a), h2(b))); }
/* 1.0 in the lanes where a = b */
__device__ __forceinline__ __half2 h_eq(uint32_t a, uint32_t b) { return __heq2(h2(a), h2(b)); }
/* max(a - 1/256, 0): the offset */
__device__ __forceinline__ uint32_t h_offset(uint32_t a)
{
    return u2(__hfma2_relu(h2(a), h2(kHOne), h2(kHNegUnit)));
}
/* learned magnitudes of capped minimums c */
__device__ __forceinline__ uint32_t h_learned(uint32_t c, uint32_t lp) { return h_of_int(learned_lut(h_to_int(c), lp)); }

template <int DM, int LS, bool WIDE, bool PO>
struct PairCheck {
    static_assert(DM <= (WIDE ? 32 : 16), "degree above the record's slots");
    using Rec = PairRec<WIDE>;
    static constexpr int S = DM;
    static constexpr int K0 = 2;
    static constexpr int K1 = S - 1 < 2 * LS + 1 ? S - 1 : 2 * LS + 1;
    uint32_t addr[S]; /* shared-memory byte addresses of the links' posteriors */
    uint32_t x[S];
    uint32_t live, inm, outm;
    uint32_t om0, omd, idxh, sgn, sgn1; /* old messages: min0, min1 - min0, index, sign bits */
    uint32_t min0, min1, sg;            /* smallest magnitudes, sign parity (bit 15 / 31) */
    uint32_t mn0, mnd, recw;            /* outgoing magnitudes with the parity's sign (set by finish), record word */

    __device__ __forceinline__ void setup(const int2* __restrict__ ent, int K, int q, int i, int j,
                                          Rec rec, uint32_t fresh, unsigned long long meta, uint32_t sbase)
    {
        const int pc = K + kQCp * i + j;
        const int pp = i ? pc - kQCp : K + kQCp * (q - 1) + j - 1;
        uint32_t lv = (uint32_t)((1ull << DM) - 1ull);
        if ((i | j) == 0)
            lv &= ~2u;
        live = lv;
        inm = (uint32_t)(meta >> 8) & 0xFFFFFFu;
        outm = (uint32_t)(meta >> 32) & 0xFFFFFFu;
        const uint32_t tj = 2u * (uint32_t)j;
#pragma unroll
        for (int k = 0; k < S; k++) {
            if (k < 2) {
                addr[k] = PO ? 0u : sbase + 2u * (uint32_t)(k == 0 ? pc : pp);
            } else {
                /* link of check j: word (j - a) mod 360 of the group, as min(u, u + 720)
                 * over unsigned byte offsets u = 2 j - 2 a */
                const int2 e = ent[k - 2];
                const uint32_t u = tj + (uint32_t)e.y;
                addr[k] = (uint32_t)e.x + __viaddmin_u32(u, 2u * kQCp, u);
            }
        }
        /* messages: zero for a lane in its first iteration */
        const uint32_t w0 = rec.x & ~fresh;
        sgn = rec.y & ~fresh;
        if constexpr (WIDE) {
            sgn1 = rec.z & ~fresh;
            idxh = (rec.w & ~fresh) | kHFour;
        } else {
            sgn1 = 0;
            idxh = ((w0 >> 12) & 0x000F000Fu) | kHFour;
        }
        om0 = h_of_int(w0 & 0x003F003Fu);
        omd = u2(__hsub2(h2(h_of_int((w0 >> 6) & 0x003F003Fu)), h2(om0)));
        min0 = min1 = kHOne;
        sg = 0;
    }

    /* minus 4 minus the old message of slot k: its magnitude with its sign, at most 31 */
    __device__ __forceinline__ uint32_t unmsg(int k) const
    {
        const uint32_t mag = u2(__hfma2(h_eq(idxh, kHFour + (uint32_t)k * 0x00010001u), h2(omd), h2(om0)));
        const int s = (k & 15) >> 1;
        const uint32_t m = ((((k < 16 ? sgn : sgn1) << ((k & 1) ? s : s + 8)) & kHSign) ^ mag);
        return u2(__hsub2(h2(kHNegFour), __hmin2(h2(m), h2(kH31))));
    }

    __device__ __forceinline__ void fold(uint32_t a)
    {
        min1 = h_min(min1, h_max(min0, a));
        min0 = h_min(min0, a);
    }

    template <bool LEV>
    __device__ __forceinline__ void read_all(uint32_t r0, uint32_t r1)
    {
        const uint32_t shared = inm | outm;
        auto slot = [&](int k) {
            const uint32_t m = unmsg(k);
            const uint32_t raw = PO && k < 2 ? (k == 0 ? r0 : r1) : lds16(addr[k]);
            uint32_t v = h_input(raw, idxh, m);
            const bool maybe_shared = LEV && k >= K0 && k <= K1;
            if (k == 1) { /* a slot that can be absent: above every minimum, positive */
                v = ((live >> k) & 1u) ? v : kHOne;
            }
            x[k] = maybe_shared && ((inm >> k) & 1u) ? m : v; /* a late slot waits for its level */
            const bool out = maybe_shared && ((shared >> k) & 1u);
            sg ^= out ? 0u : v;
            return out ? kHOne : v;
        };
#pragma unroll
        for (int k = 0; k + 1 < S; k += 2) {
            const uint32_t a = h_abs(slot(k)), b = h_abs(slot(k + 1));
            const uint32_t lo = h_min(a, b), hi = h_max(a, b);
            min1 = __vimin3_s16x2(h_max(min0, lo), min1, hi); /* halves that are not negative order as integers */
            min0 = h_min(min0, lo);
        }
        if (S & 1)
            fold(h_abs(slot(S - 1)));
    }

    __device__ __forceinline__ uint32_t smallest() const { return min0; }

    __device__ __forceinline__ void fold_shared(int k, bool use)
    {
        fold(use ? h_abs(x[k]) : kHOne);
        sg ^= use ? x[k] : 0u;
    }

    __device__ __forceinline__ void idle(uint32_t sbase)
    {
#pragma unroll
        for (int k = 0; k < S; k++) {
            addr[k] = sbase;
            x[k] = 0;
        }
        live = inm = outm = 0;
        om0 = omd = sgn = sgn1 = 0;
        idxh = kHFour;
        min0 = min1 = kHOne;
        sg = mn0 = mnd = recw = 0;
    }

    __device__ __forceinline__ void finish(bool learned, uint32_t lp)
    {
        const uint32_t c0 = h_min(min0, kH127), c1 = h_min(min1, kH127);
        const uint32_t m0 = learned ? h_learned(c0, lp) : h_offset(c0);
        const uint32_t m1 = learned ? h_learned(c1, lp) : h_offset(c1);
        mn0 = m0 ^ (sg & kHSign);
        mnd = u2(__hsub2(h2(m1), h2(m0))) ^ (sg & kHSign);
        /* per lane min0 (6 bits) | min1 << 6, magnitudes capped at 32 */
        recw = h_to_int(h_min(m0, kH32)) | (h_to_int(h_min(m1, kH32)) << 6);
    }

    __device__ __forceinline__ void write_rest(Rec* __restrict__ dst, uint32_t& o0, uint32_t& o1)
    {
        const uint32_t wm = live & ~outm;
        uint32_t nsg = 0, nsg1 = 0;
        /* the index in chains of about seven slots, the highest found */
        constexpr int CH = (S + 6) / 7;
        __half2 idxs[CH];
#pragma unroll
        for (int q = 0; q < CH; q++)
            idxs[q] = h2(kHFour);
#pragma unroll
        for (int k = 0; k < S; k++) {
            const __half2 f = h_eq(h_abs(x[k]), min0);
            const uint32_t m = u2(__hfma2(f, h2(mnd), h2(mn0))) ^ (x[k] & kHSign);
            const uint32_t nv = h_output(x[k], m);
            __half2& idx = idxs[k % CH];
            idx = __hfma2(f, __hsub2(h2(kHFour + (uint32_t)k * 0x00010001u), idx), idx);
            if (PO && k < 2)
                (k == 0 ? o0 : o1) = nv;
            else if (k > K1 && k != 1)
                sts16(addr[k], nv); /* every slot past K1 is a link written here */
            else if ((wm >> k) & 1u)
                sts16(addr[k], nv);
            if ((k & 1) || k == S - 1) {
                /* the signs of two slots in one permute */
                const int e = k & ~1;
                const uint32_t p = (k & 1) ? prmt(x[e], x[k], 0xFBD9) : prmt(x[e], 0, 0xFBD9);
                (k < 16 ? nsg : nsg1) |= p & (0x01010101u << (7 - ((e & 15) >> 1)));
            }
        }
        uint32_t nidx = u2(idxs[0]);
#pragma unroll
        for (int q = 1; q < CH; q++)
            nidx = __vmaxs2(nidx, u2(idxs[q]));
        /* the outgoing signs: each value's sign flipped where the parity is odd */
        const uint32_t pm = lmask(sg);
        nsg ^= pm;
        if constexpr (WIDE) {
            nsg1 ^= pm;
            __stcg(dst, make_uint4(recw, nsg, nsg1, nidx & 0x001F001Fu));
        } else {
            __stcg(dst, make_uint2(recw | (nidx & 0x000F000Fu) << 12, nsg));
        }
    }

    /* shared links, see level_step */
    static __device__ __forceinline__ uint32_t none() { return kHOne; }
    __device__ __forceinline__ uint32_t value(uint32_t raw, uint32_t m) const { return h_input(raw, idxh, m); }
    template <bool LEARNED>
    static __device__ __forceinline__ uint32_t inner_of(uint32_t smallest)
    {
        return h_min(smallest, kH127);
    }
    template <bool LEARNED>
    static __device__ __forceinline__ uint32_t mag(uint32_t v)
    {
        return h_abs(v);
    }
    template <bool LEARNED>
    __device__ __forceinline__ uint32_t updated(int k, uint32_t inner, uint32_t others, uint32_t sign, uint32_t lp) const
    {
        const uint32_t r = h_min(inner, others);
        const uint32_t m = LEARNED ? h_learned(r, lp) : h_offset(r);
        return h_output(x[k], m ^ ((sg ^ sign) & kHSign));
    }
    static __device__ __forceinline__ uint32_t smaller(uint32_t a, uint32_t b) { return h_min(a, b); }
};

struct PairFrame {
    uint16_t* post;
    const int2* ent; /* (shared byte address of the link group's first word, -2 a) */
    const uint16_t* eoff;
    /* parity out of shared memory (PO kernels): the posterior word of
     * parity bit (i, j) is gpar[360 i + j] (global, this CTA's slab) for
     * i < q - 1 and wrap[j] (shared) for the last layer */
    uint16_t* gpar;
    uint16_t* wrap;
};

__device__ __forceinline__ size_t a16p(size_t v) { return (v + 15) & ~(size_t)15; }

template <bool PO>
__device__ PairFrame stage_pair(const DevCode& c, char* smem, uint16_t* gpar)
{
    PairFrame f;
    f.post = (uint16_t*)smem;
    size_t off = a16p(2 * (size_t)(PO ? c.K : c.N));
    f.gpar = gpar;
    f.wrap = nullptr;
    if (PO) {
        f.wrap = (uint16_t*)(smem + off);
        off += a16p(2 * (size_t)kQCp);
    }
    int2* ent = (int2*)(smem + off);
    off += a16p(sizeof(int2) * c.nent);
    uint16_t* eoff = (uint16_t*)(smem + off);
    /* entries (360 g - a, a) as (shared byte address of group g's first
     * posterior word, -2 a): the link of check j is word (j - a) mod 360 of
     * the group, at byte offset min(u, u + 720), u = 2 j - 2 a unsigned */
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(f.post);
    for (int k = threadIdx.x; k < c.nent; k += blockDim.x) {
        const int2 e = c.ent[k];
        ent[k] = make_int2((int)(sbase + 2u * (uint32_t)(e.x + e.y)), -2 * e.y);
    }
    for (int k = threadIdx.x; k <= c.q; k += blockDim.x)
        eoff[k] = c.eoff[k];
    f.ent = ent;
    f.eoff = eoff;
    return f;
}

/* Byte `h` of the posterior word of parity bit (ii, jj) */
template <bool PO>
__device__ __forceinline__ uint8_t* parity_byte(const DevCode& c, const PairFrame& fr, uint32_t ii, uint32_t jj, int h)
{
    if (!PO)
        return (uint8_t*)fr.post + 2 * (c.K + kQCp * ii + jj) + h;
    return ii + 1 < (uint32_t)c.q ? (uint8_t*)fr.gpar + 2 * (kQCp * ii + jj) + h : (uint8_t*)fr.wrap + 2 * jj + h;
}

constexpr uint32_t kBias = 0x80808080u; /* posterior bytes are P + 128 */

/* Frame f's LLRs into byte `h` of every posterior word (f < 0: the all-zero
 * codeword at full confidence, which passes every check). */
template <bool PO>
__device__ void load_lane(const DevCode& c, const PairFrame& fr, const int8_t* __restrict__ src, int h)
{
    uint8_t* b = (uint8_t*)fr.post + h;
    const int t = threadIdx.x;
    if (!src) {
        for (int v = t; v < c.K; v += blockDim.x)
            b[2 * v] = 255;
        for (int k = t; k < c.R; k += blockDim.x)
            *parity_byte<PO>(c, fr, k / kQCp, k % kQCp, h) = 255;
        return;
    }
    if (((uintptr_t)src & 7) == 0) {
        const uint2* s8 = (const uint2*)src;
        for (int u = t; u < c.K / 8; u += blockDim.x) {
            uint2 w = __ldcs(s8 + u);
            w.x ^= kBias;
            w.y ^= kBias;
#pragma unroll
            for (int r = 0; r < 8; r++)
                b[2 * (8 * u + r)] = (uint8_t)((r < 4 ? w.x : w.y) >> (8 * (r & 3)));
        }
        const uint32_t qm = 0xFFFFFFFFu / (uint32_t)c.q + 1u;
        for (int u = t; u < c.R / 8; u += blockDim.x) {
            uint2 w = __ldcs(s8 + c.K / 8 + u);
            w.x ^= kBias;
            w.y ^= kBias;
#pragma unroll
            for (int r = 0; r < 8; r++) {
                const uint32_t k = 8u * u + r;
                const uint32_t jj = __umulhi(k, qm), ii = k - jj * c.q;
                *parity_byte<PO>(c, fr, ii, jj, h) = (uint8_t)((r < 4 ? w.x : w.y) >> (8 * (r & 3)));
            }
        }
    } else {
        for (int v = t; v < c.K; v += blockDim.x)
            b[2 * v] = (uint8_t)(src[v] ^ 0x80);
        for (int k = t; k < c.R; k += blockDim.x)
            *parity_byte<PO>(c, fr, k % c.q, k / c.q, h) = (uint8_t)(src[c.K + k] ^ 0x80);
    }
}

/* Syndrome of both lanes: bit h of the result set if lane h fails.  Thread
 * t checks column t % 360 of every other layer; the scan stops once both
 * lanes have failed.  The result is the OR over all layers, so the scan may
 * start anywhere: it starts at a layer where the previous scan found a
 * failure (srow[0], fixed during a scan; srow[1] collects a failing layer),
 * which a frame that still fails usually fails again. */
/* The posterior words of the two parity bits of check (i, j): its own and
 * the previous one (for check (0, 0), none: a positive stand-in) */
template <bool PO>
__device__ __forceinline__ void parity_words(const DevCode& c, const PairFrame& fr, int i, int j, uint32_t& pc,
                                             uint32_t& pp)
{
    if (PO) {
        pc = i + 1 < c.q ? fr.gpar[kQCp * i + j] : fr.wrap[j];
        pp = i ? fr.gpar[kQCp * (i - 1) + j] : (j ? fr.wrap[j - 1] : 0x8181u);
    } else {
        pc = fr.post[c.K + kQCp * i + j];
        pp = i ? fr.post[c.K + kQCp * (i - 1) + j] : (j ? fr.post[c.K + kQCp * (c.q - 1) + j - 1] : 0x8181u);
    }
}

template <bool PO>
__device__ int syndrome_pair(const DevCode& c, const PairFrame& fr, volatile int* sflag, volatile int* srow)
{
    const int t = threadIdx.x;
    const int nh = blockDim.x / kQCp; /* threads per column */
    const int i0 = srow[0];
    int fail = 0;
    if (t < nh * kQCp) {
        const int j = t % kQCp, h0 = t / kQCp;
        /* parity words are loaded D rows ahead (global memory in PO kernels) */
        constexpr int D = 4;
        auto row = [&](int k) { return k + i0 < c.q ? k + i0 : k + i0 - c.q; };
        uint32_t bc[D], bp[D];
#pragma unroll
        for (int d = 0; d < D; d++) {
            bc[d] = bp[d] = 0;
            if (h0 + d * nh < c.q)
                parity_words<PO>(c, fr, row(h0 + d * nh), j, bc[d], bp[d]);
        }
        bool stop = false;
        for (int k0 = h0; k0 < c.q && !stop; k0 += D * nh) {
#pragma unroll
            for (int d = 0; d < D; d++) {
                const int k = k0 + d * nh;
                if (k >= c.q || *sflag == 3) {
                    stop = true;
                    break;
                }
                const int i = row(k);
                const uint32_t pc = bc[d], pp = bp[d];
                if (k + D * nh < c.q)
                    parity_words<PO>(c, fr, row(k + D * nh), j, bc[d], bp[d]);
                /* bit 7 of a byte is set for a value that is not negative, and a byte is
                 * not 0x80 (a value not zero) if its low bits are not zero or bit 7 is clear */
                auto nonzero = [](uint32_t w) { return ((w & 0x7F7Fu) + 0x7F7Fu) | ~w; };
                uint32_t par = pc ^ pp, nz = nonzero(pc) & nonzero(pp);
                const int e0 = fr.eoff[i], e1 = fr.eoff[i + 1];
                for (int e = e0; e < e1; e++) {
                    const int2 en = fr.ent[e];
                    const uint32_t u = 2u * (uint32_t)j + (uint32_t)en.y;
                    const uint32_t w = lds16((uint32_t)en.x + __viaddmin_u32(u, 2u * kQCp, u));
                    par ^= w;
                    nz &= nonzero(w);
                }
                /* the bits that are not set count the negative values: all links less the set ones */
                const uint32_t bad = (((e1 - e0) & 1) ? ~par : par) | ~nz;
                const int f = ((bad >> 7) & 1) | ((bad >> 14) & 2);
                if (f & ~fail) {
                    fail |= f;
                    atomicOr((int*)sflag, f);
                    srow[1] = i;
                }
            }
        }
    }
    __syncthreads();
    const int r = *sflag;
    if (t == 0)
        srow[0] = srow[1];
    __syncthreads();
    return r;
}

/*
 * The step of a wavefront level, on whole warps: the checks of the level
 * (mine) read their late slots (late: any level but the first) and write the
 * posteriors that later levels read (early slots).  A level waits for the one
 * before it, so the step is kept to the chain from a late slot's posterior to
 * an early slot's: the message to a shared slot has the magnitude of the
 * smallest other link, min(inner, the other shared slots), where `inner`, the
 * smallest of the links no other check of the layer shares, capped, is known
 * before the first level, and the sign of the others' signs.  The
 * node's minimums take the shared slots after the last level (fold_shared).
 * Shared links come first in every layer (codes.cpp), so they are among slots
 * 2 .. KE: two for KE = 3, three or four for KE = 5, and so on.
 * lp: the check's learned class table (learned kernels).
 *
 * Bound by that chain's latency, 3 to 4 warps a level between CTA barriers: it
 * took the node's whole finish (minimums, both candidates, the index) and every
 * shared slot's update before.  With two, four, six and more slots compiled
 * apart, us of the GPU per frame-iteration: normal 3/5 0.400 -> 0.376, 1/3
 * 0.426 -> 0.378, 5/6 0.407 -> 0.340, 8/9 0.360 -> 0.264, short 1/2 0.095 ->
 * 0.086, 3/5 0.181 -> 0.143, 5/6 0.182 -> 0.157 (all with the node on 16-bit
 * integers).  The forms are written out: one form over every slot's test that
 * takes the two smallest left normal 9/10 at 0.342 and 4/5 at 0.294, which run
 * at 0.250 and 0.261.
 */
template <int KE, class Ck>
__device__ __forceinline__ void read_late(Ck& ck, bool mine)
{
    const uint32_t im = mine ? ck.inm : 0u;
#pragma unroll
    for (int k = Ck::K0; k <= KE; k++) {
        const uint32_t v = ck.value(lds16(ck.addr[k]), ck.x[k]);
        ck.x[k] = (im >> k) & 1u ? v : ck.x[k];
    }
}

template <int KE, bool LEARNED, class Ck>
__device__ __forceinline__ void level_step(Ck& ck, uint32_t inner, bool mine, bool late, uint32_t lp)
{
    const uint32_t NONE = Ck::none(); /* above every magnitude */
    const uint32_t im = mine ? ck.inm : 0u, om = mine ? ck.outm : 0u, sh = ck.inm | ck.outm;
    auto read = [&](int k) {
        if (late) {
            const uint32_t v = ck.value(lds16(ck.addr[k]), ck.x[k]);
            ck.x[k] = (im >> k) & 1u ? v : ck.x[k];
        }
        return Ck::template mag<LEARNED>(ck.x[k]);
    };
    /* slot k, the smallest magnitude and the sign of the other shared slots */
    auto write = [&](int k, uint32_t others, uint32_t sign) {
        const uint32_t nv = ck.template updated<LEARNED>(k, inner, others, sign, lp);
        if ((om >> k) & 1u)
            sts16(ck.addr[k], nv);
    };
    if constexpr (KE < 3) {
        return; /* no two links of a layer are shared */
    } else if constexpr (KE == 3) {
        const uint32_t a = read(2), b = read(3);
        write(2, b, ck.x[3]);
        write(3, a, ck.x[2]);
    } else if constexpr (KE == 5) { /* three or four */
        const bool four = (sh >> 5) & 1u;
        const uint32_t a = read(2), b = read(3), c = read(4), r5 = read(5);
        const uint32_t d = four ? r5 : NONE;
        const uint32_t ab = Ck::smaller(a, b), cd = Ck::smaller(c, d);
        const uint32_t sab = ck.x[2] ^ ck.x[3], s5 = four ? ck.x[5] : 0u, scd = ck.x[4] ^ s5;
        write(2, Ck::smaller(b, cd), ck.x[3] ^ scd);
        write(3, Ck::smaller(a, cd), ck.x[2] ^ scd);
        write(4, Ck::smaller(ab, d), sab ^ s5);
        write(5, Ck::smaller(ab, c), sab ^ ck.x[4]);
    } else if constexpr (KE == 7) { /* five or six */
        const bool six = (sh >> 7) & 1u;
        const uint32_t a = read(2), b = read(3), c = read(4), d = read(5), e = read(6), r7 = read(7);
        const uint32_t f = six ? r7 : NONE;
        const uint32_t ab = Ck::smaller(a, b), cd = Ck::smaller(c, d), ef = Ck::smaller(e, f);
        const uint32_t abcd = Ck::smaller(ab, cd), abef = Ck::smaller(ab, ef), cdef = Ck::smaller(cd, ef);
        const uint32_t sab = ck.x[2] ^ ck.x[3], scd = ck.x[4] ^ ck.x[5], s7 = six ? ck.x[7] : 0u, sef = ck.x[6] ^ s7;
        write(2, Ck::smaller(b, cdef), ck.x[3] ^ scd ^ sef);
        write(3, Ck::smaller(a, cdef), ck.x[2] ^ scd ^ sef);
        write(4, Ck::smaller(d, abef), ck.x[5] ^ sab ^ sef);
        write(5, Ck::smaller(c, abef), ck.x[4] ^ sab ^ sef);
        write(6, Ck::smaller(f, abcd), s7 ^ sab ^ scd);
        write(7, Ck::smaller(e, abcd), ck.x[6] ^ sab ^ scd);
    } else if constexpr (KE == 9) { /* seven or eight */
        const bool eight = (sh >> 9) & 1u;
        const uint32_t a = read(2), b = read(3), c = read(4), d = read(5), e = read(6), f = read(7), g = read(8),
                       r9 = read(9);
        const uint32_t h = eight ? r9 : NONE;
        const uint32_t ab = Ck::smaller(a, b), cd = Ck::smaller(c, d), ef = Ck::smaller(e, f), gh = Ck::smaller(g, h);
        const uint32_t abcd = Ck::smaller(ab, cd), efgh = Ck::smaller(ef, gh);
        const uint32_t s9 = eight ? ck.x[9] : 0u, s25 = ck.x[2] ^ ck.x[3] ^ ck.x[4] ^ ck.x[5],
                       s69 = ck.x[6] ^ ck.x[7] ^ ck.x[8] ^ s9, all = s25 ^ s69;
        uint32_t rest = Ck::smaller(cd, efgh);
        write(2, Ck::smaller(b, rest), all ^ ck.x[2]);
        write(3, Ck::smaller(a, rest), all ^ ck.x[3]);
        rest = Ck::smaller(ab, efgh);
        write(4, Ck::smaller(d, rest), all ^ ck.x[4]);
        write(5, Ck::smaller(c, rest), all ^ ck.x[5]);
        rest = Ck::smaller(gh, abcd);
        write(6, Ck::smaller(f, rest), all ^ ck.x[6]);
        write(7, Ck::smaller(e, rest), all ^ ck.x[7]);
        rest = Ck::smaller(ef, abcd);
        write(8, Ck::smaller(h, rest), all ^ ck.x[8]);
        write(9, Ck::smaller(g, rest), all ^ ck.x[9]);
    } else { /* nine to twelve (or, in a kernel without the forms above, fewer) */
        uint32_t r[12], sx[12];
#pragma unroll
        for (int n = 0; n < 12; n++) {
            const int k = 2 + n;
            r[n] = NONE;
            sx[n] = 0;
            if (k <= KE) {
                const bool is = n < 5 || ((sh >> k) & 1u);
                const uint32_t v = read(k);
                r[n] = is ? v : NONE;
                sx[n] = is ? ck.x[k] : 0u;
            }
        }
        constexpr bool MORE = KE > 9;
        const uint32_t ab = Ck::smaller(r[0], r[1]), cd = Ck::smaller(r[2], r[3]), ef = Ck::smaller(r[4], r[5]),
                       gh = Ck::smaller(r[6], r[7]);
        const uint32_t ij = MORE ? Ck::smaller(r[8], r[9]) : NONE, kl = MORE ? Ck::smaller(r[10], r[11]) : NONE;
        const uint32_t ijkl = MORE ? Ck::smaller(ij, kl) : NONE;
        auto with = [&](uint32_t v) { return MORE ? Ck::smaller(v, ijkl) : v; };
        const uint32_t abcd = Ck::smaller(ab, cd), efgh = Ck::smaller(ef, gh);
        const uint32_t lo = with(efgh), hi = with(abcd);
        uint32_t all = sx[0] ^ sx[1] ^ sx[2] ^ sx[3] ^ sx[4] ^ sx[5] ^ sx[6] ^ sx[7];
        if (MORE)
            all ^= sx[8] ^ sx[9] ^ sx[10] ^ sx[11];
        auto pair = [&](int n, uint32_t rest) { /* rest: the other pairs */
            if (2 + n <= KE)
                write(2 + n, Ck::smaller(r[n + 1], rest), all ^ ck.x[2 + n]);
            if (3 + n <= KE)
                write(3 + n, Ck::smaller(r[n], rest), all ^ ck.x[3 + n]);
        };
        pair(0, Ck::smaller(cd, lo));
        pair(2, Ck::smaller(ab, lo));
        pair(4, Ck::smaller(gh, hi));
        pair(6, Ck::smaller(ef, hi));
        if constexpr (MORE) {
            const uint32_t all8 = Ck::smaller(abcd, efgh);
            pair(8, Ck::smaller(kl, all8));
            pair(10, Ck::smaller(ij, all8));
        }
    }
}

/*
 * Layer i of the phased schedule.  Every check reads its links that no
 * other check of the layer shares, or that no earlier check writes (a
 * full-occupancy pass); then, level by level, the checks of the level read
 * their late links and write the posteriors that later checks of the layer
 * read (level_step); a last full pass folds the shared links into the
 * minimums and writes every other posterior and the messages.  The
 * reference's in-order semantics only constrain the bits two checks of a
 * layer share, so the wavefront levels carry just those links.  Unlevelled
 * layers take one pass.
 */
template <int DM, int LS, bool WIDE, bool LEARNED, bool PO>
__device__ __forceinline__ void layer_pair(const PairFrame& fr, const DevCode& c, const int2* ent, int i, int nlev,
                                           PairRec<WIDE> rec, unsigned long long meta, uint32_t fresh,
                                           PairRec<WIDE>* __restrict__ msg, uint32_t r0, uint32_t r1,
                                           uint32_t& o0, uint32_t& o1)
{
    const int t = threadIdx.x;
    const bool active = t < kQCp;
    const int j = t;
    /* the check's learned class table (an index into s_learn_lut) */
    auto lclass = [&]() {
        return LEARNED ? 128u * (uint32_t)s_learn_cls[DM - ((i | j) == 0)] : 0u;
    };
    using Ck = PairCheck<DM, LS, WIDE, PO>;
    Ck ck;
    if (active) {
        ck.setup(ent, c.K, c.q, i, j, rec, fresh, meta,
                 (uint32_t)__cvta_generic_to_shared(fr.post));
        if (LS > 0 && nlev > 1)
            ck.template read_all<true>(r0, r1);
        else
            ck.template read_all<false>(r0, r1);
    } else {
        ck.idle((uint32_t)__cvta_generic_to_shared(fr.post));
    }
    uint32_t lp = 0;
    if (active)
        lp = lclass();
    if (LS > 0 && nlev > 1) {
        /* a level step runs on every warp that holds a check of the level,
         * with all its lanes; the other checks keep their state.  KE: the
         * last slot that can be late or early in this warp (most
         * layers share one pair of links: link slots 2 and 3 only) */
        const int lev = active ? (int)(meta & 0xFF) : -1;
        const uint32_t inner = Ck::template inner_of<LEARNED>(ck.smallest());
        auto steps = [&](auto ke) {
            constexpr int KE = decltype(ke)::value;
            for (int l = 0; l < nlev - 1; l++) {
                const bool mine = lev == l;
                if (__any_sync(0xFFFFFFFFu, mine))
                    level_step<KE, LEARNED>(ck, inner, mine, l > 0, lp);
                __syncthreads();
            }
            /* the last level writes nothing early and nothing waits for it */
            if (__any_sync(0xFFFFFFFFu, lev == nlev - 1))
                read_late<KE>(ck, lev == nlev - 1);
            const uint32_t sh = ck.inm | ck.outm;
#pragma unroll
            for (int k = Ck::K0; k <= KE; k++)
                ck.fold_shared(k, KE == 3 || ((sh >> k) & 1u));
        };
        constexpr int KS = Ck::K1 > 3 ? 3 : Ck::K1, KM = Ck::K1 > 5 ? 5 : Ck::K1,
                      KL = Ck::K1 > 7 ? 7 : Ck::K1, KN = Ck::K1 > 9 ? 9 : Ck::K1;
        const uint32_t lm = __reduce_or_sync(0xFFFFFFFFu, ck.inm | ck.outm);
        if (KS == Ck::K1 || (lm >> (KS + 1)) == 0)
            steps(std::integral_constant<int, KS>());
        else if (KM == Ck::K1 || (lm >> (KM + 1)) == 0)
            steps(std::integral_constant<int, KM>());
        else if (KL == Ck::K1 || (lm >> (KL + 1)) == 0)
            steps(std::integral_constant<int, KL>());
        else if (KN == Ck::K1 || (lm >> (KN + 1)) == 0)
            steps(std::integral_constant<int, KN>());
        else
            steps(std::integral_constant<int, Ck::K1>());
    }
    if (active) {
        ck.finish(LEARNED, lp);
        ck.write_rest(msg + kQCp * i + j, o0, o1);
    }
    __syncthreads();
}

/* Layer i with the exact-degree node of its count, one of A, A + STEP .. B */
template <int A, int B, int STEP, int LS, bool WIDE, bool LEARNED, bool PO>
__device__ __forceinline__ void layer_of_count(const PairFrame& fr, const DevCode& c, const int2* ent, int i, int cnt, int nlev,
                                               PairRec<WIDE> rec, unsigned long long meta, uint32_t fresh,
                                               PairRec<WIDE>* __restrict__ msg, uint32_t r0, uint32_t r1,
                                               uint32_t& o0, uint32_t& o1)
{
    if (A == B || cnt == A)
        layer_pair<A + 2, LS, WIDE, LEARNED, PO>(fr, c, ent, i, nlev, rec, meta, fresh, msg, r0, r1, o0, o1);
    else if constexpr (A < B)
        layer_of_count<A + STEP, B, STEP, LS, WIDE, LEARNED, PO>(fr, c, ent, i, cnt, nlev, rec, meta, fresh, msg, r0, r1,
                                                                 o0, o1);
}

/* One decoding iteration: the layers in order; each layer's messages and
 * level metadata are fetched one layer ahead.  The kernel is compiled for
 * the two information-link counts A <= B of its codes (exact-degree check
 * nodes), or, with EVERY, for every count from A to B. */
template <int A, int B, int EVERY, int LS, bool LEARNED, bool PO>
__device__ void iterate_pair(const DevCode& c, const PairFrame& fr, void* msgv, uint32_t fresh, int lA, int lB)
{
    constexpr bool WIDE = B + 2 > 16;
    using Rec = PairRec<WIDE>;
    Rec* __restrict__ msg = (Rec*)msgv;
    const int t = threadIdx.x;
    const int j = t;
    const bool active = t < kQCp;
    /* the next layer's levels, read a layer ahead: read in their own layer, every warp
     * waited for them at its start (normal 2/3 0.279 -> 0.242 us per frame-iteration,
     * 1/2 0.264 -> 0.223, together with entries at A i where A = B) */
    int nl = c.nlev[0];
    Rec rn{};
    unsigned long long mn = 0;
    /* PO: the words of parity bits (i, j) and (i + 1, j) for layers i and
     * i + 1 (loaded two layers ahead), and of (i - 1, j), which the previous
     * layer of this thread wrote */
    uint32_t pnext = 0, pnext2 = 0, carry = 0;
    if (LEARNED) {
        /* this iteration's learned magnitudes: lane A's row lA, lane B's lB */
        for (int e = t; e < 2 * kLearnClasses * 128; e += blockDim.x) {
            const int h = e / (kLearnClasses * 128), k = (e / 128) % kLearnClasses;
            s_learn_lut[e] = (uint8_t)min(learned_mag(e % 128, s_learn_tab[(h ? lB : lA) + k]), 255);
        }
        __syncthreads();
    }
    if (active) {
        rn = __ldcg(msg + j);
        mn = __ldg(c.lmeta + j);
        if (PO && c.q > 1)
            pnext = fr.gpar[j];
        if (PO && c.q > 2)
            pnext2 = fr.gpar[kQCp + j];
    }
    for (int i = 0; i < c.q; i++) {
        const Rec rec = rn;
        const unsigned long long meta = mn;
        uint32_t r0 = 0, r1 = 0, o0 = 0, o1 = 0;
        if (active && i + 1 < c.q) {
            rn = __ldcg(msg + kQCp * (i + 1) + j);
            mn = __ldg(c.lmeta + kQCp * (i + 1) + j);
        }
        if (PO && active) {
            r0 = i + 1 < c.q ? pnext : fr.wrap[j];
            pnext = pnext2;
            if (i + 3 < c.q)
                pnext2 = fr.gpar[kQCp * (i + 2) + j];
            r1 = i ? carry : (j ? fr.wrap[j - 1] : 0u);
        }
        const int first = A == B ? A * i : fr.eoff[i];
        const int cnt = A == B ? A : fr.eoff[i + 1] - first;
        const int2* ent = fr.ent + first;
        const int nlev = nl;
        nl = c.nlev[i + 1 < c.q ? i + 1 : i];
        layer_of_count<A, B, EVERY ? 1 : B - A, LS, WIDE, LEARNED, PO>(fr, c, ent, i, cnt, nlev, rec, meta, fresh, msg,
                                                                       r0, r1, o0, o1);
        /* (i - 1, j) is final for this iteration; (i, j) goes to the next
         * layer, or, for the last layer, to the check (0, j + 1) */
        if (PO && active) {
            if (i)
                fr.gpar[kQCp * (i - 1) + j] = (uint16_t)o1;
            else if (j)
                fr.wrap[j - 1] = (uint16_t)o1;
            if (i + 1 < c.q)
                carry = o0;
            else
                fr.wrap[j] = (uint16_t)o0;
        }
    }
    if (PO)
        __syncthreads(); /* the last layer's wrap words before the syndrome reads them */
}

static __device__ void store_lane(const DevCode& c, const PairFrame& fr, int h, uint8_t* __restrict__ dst)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const uint8_t* b = (const uint8_t*)fr.post + h;
    const int nchunks = (c.kldpc + 31) / 32;
    for (int ch = warp; ch < nchunks; ch += nw) {
        const int v = ch * 32 + lane;
        const int x = v < c.kldpc ? b[2 * v] : 0x80;
        const unsigned m = __ballot_sync(0xFFFFFFFFu, x < 0x80);
        const unsigned rr = __byte_perm(__brev(m), 0, 0x0123);
        if (lane < 4 && 4 * ch + lane < c.nbytes)
            dst[4 * ch + lane] = (uint8_t)(rr >> (8 * lane));
    }
}

/* Group barrier of a team of M co-resident CTAs (a cooperative launch):
 * returns 1 if no member saw a failing frame, 0 if one did, -1 if the
 * barrier gave up after `limit` polls (the device error word is set to 2).
 * skip: this CTA does not arrive (a test of the time-out) and returns -1. */
static __device__ int pair_team_vote(unsigned* slot, int M, bool fail, int* err, int limit, bool skip)
{
    __shared__ int s_res;
    if (M == 1 && !skip) /* a team of one has nobody to ask */
        return fail ? 0 : 1;
    if (threadIdx.x == 0) {
        unsigned* arrive = slot;
        unsigned* fails = slot + 1;
        int res = 0;
        if (skip) {
            res = -1;
        } else {
            if (fail)
                atomicAdd(fails, 1u);
            __threadfence();
            atomicAdd(arrive, 1u);
            int spins = 0;
            while (*(volatile unsigned*)arrive < (unsigned)M) {
                if (++spins > limit) {
                    atomicExch(err, 2);
                    res = -1;
                    break;
                }
                __nanosleep(200);
            }
            __threadfence();
            if (res == 0)
                res = *(volatile unsigned*)fails == 0 ? 1 : 0;
        }
        s_res = res;
    }
    __syncthreads();
    const int r = s_res;
    __syncthreads();
    return r;
}

/* Lane state of a frame-pair CTA (shared memory): the frame and iteration
 * of each lane, the syndrome flags, the lanes to reload, the syndrome
 * scan's start rows. */
struct PairLanes {
    int frame[2], iter[2], flag, reload, row[2];
};

/* Per-frame stopping: frames stream through the two lanes independently.
 * A lane whose frame passes the syndrome check or reaches max_iter writes
 * its results and takes the next frame of the batch (the counter p.work;
 * work item k is row p.rows[k], or k), so a converged frame never waits for
 * its neighbour.  The CTA's tables are staged (fr) and its lane state
 * initialised (frames -1, both lanes to reload, flag 0, rows 0). */
template <int A, int B, int EVERY, int LS, bool PO>
__device__ __forceinline__ void stream_frames(const DecodeParams& p, const DevCode& c, const PairFrame& fr, void* msg,
                                              int lT, int nframes, PairLanes& st)
{
    int* s_frame = st.frame;
    int* s_iter = st.iter;
    int& s_flag = st.flag;
    int& s_reload = st.reload;
    int* s_row = st.row;
    const int t = threadIdx.x;
    uint32_t fresh = 0;
    for (;;) {
        /* lanes that need a frame take the next one of the batch */
        const int reload = s_reload;
        if (reload) {
            if (t == 0) {
                for (int h = 0; h < 2; h++)
                    if (reload & (1 << h)) {
                        const int f = (int)atomicAdd(p.work, 1u);
                        s_frame[h] = f < nframes ? f : -1;
                        s_iter[h] = 0;
                    }
            }
            __syncthreads();
            for (int h = 0; h < 2; h++)
                if (reload & (1 << h)) {
                    const int f = s_frame[h];
                    const int row = f < 0 ? 0 : p.rows ? p.rows[f] : f;
                    load_lane<PO>(c, fr, f >= 0 ? p.llr + (size_t)row * p.llr_stride : nullptr, h);
                    fresh |= 0xFFFFu << (16 * h);
                }
            if (t == 0)
                s_reload = 0;
            __syncthreads();
        }
        if (s_frame[0] < 0 && s_frame[1] < 0)
            break;
        const int fail = syndrome_pair<PO>(c, fr, &s_flag, s_row);
        /* lanes whose frame is done: results out, refill */
        int done = 0;
        for (int h = 0; h < 2; h++) {
            const int f = s_frame[h];
            if (f >= 0 && (!((fail >> h) & 1) || s_iter[h] >= p.max_iter)) {
                const int row = p.rows ? p.rows[f] : f;
                store_lane(c, fr, h, p.out + (size_t)row * p.out_stride);
                if (t == 0) {
                    if (p.iters)
                        p.iters[row] = s_iter[h];
                    if (p.ok)
                        p.ok[row] = (fail >> h) & 1 ? 0 : 1;
                }
                done |= 1 << h;
            }
        }
        __syncthreads();
        if (t == 0) {
            s_flag = 0;
            s_reload = done;
        }
        __syncthreads();
        if (done)
            continue; /* reload, then check the new frames first */
        if (lT)
            iterate_pair<A, B, EVERY, LS, true, PO>(c, fr, msg, fresh, learn_row(s_iter[0], lT),
                                                  learn_row(s_iter[1], lT));
        else
            iterate_pair<A, B, EVERY, LS, false, PO>(c, fr, msg, fresh, -1, -1);
        fresh = 0;
        if (t == 0) {
            s_iter[0]++;
            s_iter[1]++;
        }
        __syncthreads();
    }
}

/* PM: 0 one resident CTA per SM; 1 two (80 registers), for codes whose
 * posteriors leave room for two (short frames); 2 two, with the parity
 * posteriors out of shared memory (PO: normal frames up to rate 4/5) */
template <int A, int B, int EVERY, int LS, int PM>
__global__ void __launch_bounds__(384, PM ? 2 : 1) k_decode_pair(DecodeParams p)
{
    constexpr bool PO = PM == 2;
    extern __shared__ __align__(16) char smem[];
    __shared__ int s_lanes[sizeof(PairLanes) / sizeof(int)];
    int* s_frame = ((PairLanes*)s_lanes)->frame;
    int& s_flag = ((PairLanes*)s_lanes)->flag;
    int& s_reload = ((PairLanes*)s_lanes)->reload;
    int* s_row = ((PairLanes*)s_lanes)->row;
    const DevCode c = *p.code;
    constexpr bool WIDE = B + 2 > 16;
    void* msg = (char*)p.msg + (size_t)blockIdx.x * p.msg_stride;
    /* the parity words follow the message records in this CTA's slab */
    uint16_t* gpar = (uint16_t*)((char*)msg + (((size_t)c.R * (WIDE ? 16 : 8) + 15) & ~(size_t)15));
    const PairFrame fr = stage_pair<PO>(c, smem, gpar);
    const int lT = stage_learn(p.learn, p.learn_class, p.learn_iters);
    const int nframes = p.nframes_dev ? *p.nframes_dev : p.nframes;
    const int t = threadIdx.x;
    if (t == 0) {
        s_frame[0] = s_frame[1] = -1;
        s_flag = 0;
        s_reload = 3;
        s_row[0] = s_row[1] = 0;
    }
    __syncthreads();
    if (p.group > 0) {
        /* group stopping (the reference's batch semantics): the G frames of a
         * group run on a team of M = ceil(G / 2) CTAs, two frames each, and
         * stop together at the first syndrome that every frame passes */
        const int G = p.group, M = (G + 1) / 2;
        const int team = blockIdx.x / M, member = blockIdx.x % M;
        const int ngroups = (p.nframes + G - 1) / G;
        const int per = p.max_iter + 1, per_team = (ngroups + p.nteams - 1) / p.nteams;
        for (int g = team, k = 0; g < ngroups; g += p.nteams, k++) {
            unsigned* sync = p.team_sync + 2 * (size_t)per * ((size_t)team * per_team + k);
            const int end = min((g + 1) * G, p.nframes);
            int fr2[2];
            for (int h = 0; h < 2; h++) {
                const int f = g * G + 2 * member + h;
                fr2[h] = f < end ? f : -1;
                const int row = fr2[h] < 0 ? 0 : p.rows ? p.rows[fr2[h]] : fr2[h];
                load_lane<PO>(c, fr, fr2[h] >= 0 ? p.llr + (size_t)row * p.llr_stride : nullptr, h);
            }
            __syncthreads();
            uint32_t gfresh = 0xFFFFFFFFu;
            int it = 0;
            bool ok = true;
            for (;;) {
                const int fail = syndrome_pair<PO>(c, fr, &s_flag, s_row);
                if (t == 0)
                    s_flag = 0; /* read again only after later barriers */
                const int v = pair_team_vote(sync + 2 * it, M, fail != 0, p.err,
                                             p.wait_limit > 0 ? p.wait_limit : kDefaultWaitLimit,
                                             (int)blockIdx.x + 1 == p.skip_vote);
                ok = v == 1;
                if (v < 0 || ok || it >= p.max_iter)
                    break;
                iterate_pair<A, B, EVERY, LS, false, PO>(c, fr, msg, gfresh, -1, -1);
                gfresh = 0;
                it++;
            }
            for (int h = 0; h < 2; h++)
                if (fr2[h] >= 0) {
                    const int row = p.rows ? p.rows[fr2[h]] : fr2[h];
                    store_lane(c, fr, h, p.out + (size_t)row * p.out_stride);
                    if (t == 0) {
                        if (p.iters)
                            p.iters[row] = it;
                        if (p.ok)
                            p.ok[row] = ok ? 1 : 0;
                    }
                }
            __syncthreads();
        }
        return;
    }
    PairLanes& st = *(PairLanes*)s_lanes;
    stream_frames<A, B, EVERY, LS, PO>(p, c, fr, msg, lT, nframes, st);
}

/* Pair kernels by information-link counts (A, B): every pair of the DVB-S2,
 * S2X and T2 codes, or every count from A to B (every = 1).  LS:
 * half the shared slots the kernel carries. */
struct PairKernel {
    int a, b, every, ls, pm, threads;
    const void* fn;
};


/* The instantiated kernels, in parts (part k in ldpc_pair_k<k>.cu):
 * pair_kernel_part(k, &n) returns part k and its n entries. */
const PairKernel* pair_kernel_part(int part, int* n);
constexpr int kPairKernelParts = 6;

/* launch bounds of a residency mode: 1 CTA per SM (mode 0) or two */
#define DRXG_PAIR_KERNEL(a, b, every, ls, pm) { a, b, every, ls, pm, 384, (const void*)k_decode_pair<a, b, every, ls, pm> }

}  // namespace drxg
