/*
 * Learned (neural offset / scaled) min-sum: training kernels and parameters.
 */
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "codes.h"
#include "ldpc_device.h"

namespace drxg {

constexpr int kLearnedMaxDeg = 32;  /* links of a check node */
constexpr int kLearnedMaxClass = 8; /* check-degree classes */

/* One training or evaluation launch over nframes frames of one code. */
struct LearnedParams {
    const DevCode* code; /* device */
    int nframes;
    int iters;
    int DS;              /* message slots per check: the code's largest degree */
    const __half* llr;   /* nframes rows of llr_stride halves: unquantised 2 x LLR */
    size_t llr_stride;
    const uint8_t* bits; /* nframes rows: kldpc information bits, MSB first */
    size_t bits_stride;
    const __half* beta;  /* iters x nclass FP16 scales */
    const __half* alpha; /* iters x nclass FP16 offsets */
    int nclass;
    const int8_t* cls;   /* class of each check degree 0..32 (device) */
    float* P;            /* workspace: nframes x N posteriors */
    uint4* M;            /* nframes x R message records */
    float* gP;           /* backward: nframes x N */
    float* gM;           /* backward: nframes x DS*R (layer, slot, check) */
    float* Pck;          /* training: iters x nframes x K posteriors after each iteration (null: none) */
    float* Xck;          /* iters x nframes x DS*R extrinsic inputs (layer, slot, check) */
    float* loss;         /* iters: sums of the BCE of every iteration's output */
    float* dbeta;        /* backward: iters x nclass */
    float* dalpha;
    float loss_scale;    /* backward: d loss / d (each per-iteration BCE sum) */
    const float* loss_w; /* backward, optional: per-iteration weights of the BCE sums (device) */
    float* post;         /* forward, optional: nframes x kldpc final posteriors */
};

cudaError_t launch_learned(const LearnedParams& p, bool backward, const Code& code, cudaStream_t s);

}  // namespace drxg
