/*
 * Baseband layer on the GPU, after the BCH decoder: BBFRAME descrambling and
 * the BBHEADER check (EN 302 307-1 5.1.6, 5.2.2), with the reference's
 * results (libdvbrx/src/bb.c:46-101: drx_bb_descramble, drx_bbheader_parse),
 * so that the device hands out BBFRAMEs ready for the TS reconstruction.
 *
 * The scrambling sequence (1 + x^14 + x^15, restarted on every BBFRAME) and
 * the CRC-8 table (0xD5) are generated from the standard into bb_tables.h
 * (dvbrx_b200/tables/gen_bb.py) and live in device memory.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "../../include/dvbrx_b200.h"
#include "bb_tables.h"
#include "handle.h"

namespace drxg {

constexpr int kBbThreads = 128;

/* frames[f][i] ^= prbs[i], i < kbytes: a thread takes the 16-byte blocks at one
 * place of its rows, aligned in memory, so that full blocks move in one load
 * and one store whatever the row's own alignment; the sequence's bytes come
 * from five words, shifted by the row's offset (they stay in L1).  Bound by
 * the rows' traffic, read and written once: 4096 normal 3/5 frames (40 MB) 19
 * -> 11 us; four bytes a thread with the sequence loaded byte by byte before. */
__global__ void __launch_bounds__(kBbThreads) k_bb_descramble(uint8_t* frames, size_t stride, int kbytes,
                                                             int nframes)
{
    const int at = 16 * (blockIdx.x * blockDim.x + threadIdx.x);
    for (int f = blockIdx.y; f < nframes; f += gridDim.y) {
        uint8_t* row = frames + (size_t)f * stride;
        const int off = at - (int)((uintptr_t)row & 15); /* of the block, in the row */
        if (off >= kbytes)
            continue;
        if (off >= 0 && off + 16 <= kbytes) {
            const uint32_t* s = (const uint32_t*)g_bb_prbs + (off >> 2);
            const uint32_t sh = 8u * (off & 3);
            uint4 v = *(const uint4*)(row + off);
            const uint32_t s0 = s[0], s1 = s[1], s2 = s[2], s3 = s[3], s4 = s[4];
            v.x ^= __funnelshift_r(s0, s1, sh);
            v.y ^= __funnelshift_r(s1, s2, sh);
            v.z ^= __funnelshift_r(s2, s3, sh);
            v.w ^= __funnelshift_r(s3, s4, sh);
            *(uint4*)(row + off) = v;
        } else {
            for (int k = max(off, 0); k < off + 16 && k < kbytes; k++)
                row[k] ^= g_bb_prbs[k];
        }
    }
}

/* BBHEADER of every frame: 0 valid, 1 valid in DVB-T2 High Efficiency Mode
 * (the CRC XOR 1, for a TS without ISSY), -1 invalid (bb.c:69-101) */
__global__ void __launch_bounds__(kBbThreads) k_bbheader(const uint8_t* frames, size_t stride, int8_t* status,
                                                        int nframes)
{
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nframes)
        return;
    const uint8_t* h = frames + (size_t)f * stride;
    uint8_t b[10];
#pragma unroll
    for (int k = 0; k < 10; k++)
        b[k] = h[k];
    uint8_t c = 0;
#pragma unroll
    for (int k = 0; k < 9; k++)
        c = g_bb_crc8[c ^ b[k]];
    int st = 0;
    if (c != b[9]) {
        if ((uint8_t)(c ^ 1) != b[9] || b[0] >> 6 != 3 || (b[0] & 0x08) || b[2] || b[3] || b[6])
            st = -1;
        else
            st = 1;
    }
    if (st >= 0) {
        const int dfl = b[4] << 8 | b[5], syncd = b[7] << 8 | b[8];
        if (dfl % 8 || dfl > DRXG_KBCH_MAX_BYTES * 8 - 80)
            st = -1;
        else if (b[0] >> 6 == 3 && (syncd > dfl || syncd % 8))
            st = -1;
    }
    status[f] = (int8_t)st;
}

}  // namespace drxg

using namespace drxg;

extern "C" {

int drx_bb_descramble_device(uint8_t* frames, size_t stride, int kbch_bytes, int nframes, void* stream)
{
    if (nframes <= 0)
        return 0;
    if (!frames || kbch_bytes < 0 || kbch_bytes > DRXG_KBCH_MAX_BYTES || stride < (size_t)kbch_bytes) {
        set_error("drx_bb_descramble_device: bad arguments");
        return -1;
    }
    /* blocks that rows of any alignment touch: the row's bytes and up to 15 before it */
    const int gx = ((kbch_bytes + 15) / 16 + 1 + kBbThreads - 1) / kBbThreads;
    const dim3 grid(gx, std::min(nframes, 4096));
    k_bb_descramble<<<grid, kBbThreads, 0, (cudaStream_t)stream>>>(frames, stride, kbch_bytes, nframes);
    return cuda_check(cudaGetLastError(), "descrambler launch") ? 0 : -1;
}

int drx_bbheader_check_device(const uint8_t* frames, size_t stride, int8_t* status, int nframes, void* stream)
{
    if (nframes <= 0)
        return 0;
    if (!frames || !status || stride < 10) {
        set_error("drx_bbheader_check_device: bad arguments");
        return -1;
    }
    k_bbheader<<<(nframes + kBbThreads - 1) / kBbThreads, kBbThreads, 0, (cudaStream_t)stream>>>(frames, stride,
                                                                                               status, nframes);
    return cuda_check(cudaGetLastError(), "BBHEADER check launch") ? 0 : -1;
}

}  // extern "C"
