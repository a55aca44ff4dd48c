// Decode of many codec frames in one pass, fp32: the reference's QwenCodecDecoder.forward outside a streaming context
// (src/vui/qwen_codec.py:1199-1215): zero left padding, causal attention over the whole input.  Frame by frame (codec_kernels.cuh)
// every frame reads all 423 MB of weights; here a matrix is read once for all frames and the work, 5 GFLOP a frame, goes to the
// tensor cores as split GEMMs (split_gemm.cuh).  This file holds the two ends: codebook lookup and the last convolution.
#pragma once
#include "split_ops.cuh"

namespace vuib_codec_batch {

using vuis::SgPlanes;

struct BEmbedArgs {
    const long long* codes;      // [n_q][T]
    int n_q, T;
    const float* table[16];      // codebook q: (2048, 256); q = 0 semantic, 1.. acoustic
    SgPlanes o;                  // 512 channels: sum of the semantic code vectors, sum of the acoustic ones
    int* flag;                   // set to flag_bad by a code outside [0, 2048)
    int flag_bad;
    int* whole;                  // set to T
};

// SplitResidualVQ.decode's sums (qwen_codec.py:231-238), in codebook order.  A CTA takes one frame.
static __global__ void __launch_bounds__(256) k_bembed(BEmbedArgs a) {
    __shared__ __align__(16) float s[512];
    vuis::sg_pdl_wait();
    vuis::sg_pdl_launch();
    const int t = blockIdx.x, c = threadIdx.x;
    long long code[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) code[q] = q < a.n_q ? __ldg(a.codes + (long long)q * a.T + t) : 0;
    bool bad = false;
#pragma unroll
    for (int q = 0; q < 16; ++q)
        if (code[q] < 0 || code[q] >= 2048) { bad = true; code[q] = code[q] < 0 ? 0 : 2047; }
    if (bad && c == 0) atomicOr(a.flag, a.flag_bad);
    float v[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) v[q] = q < a.n_q ? __ldg(a.table[q] + code[q] * 256 + c) : 0.f;
    float acq = 0.f;
#pragma unroll
    for (int q = 1; q < 16; ++q) acq += v[q];
    s[c] = v[0];
    s[256 + c] = acq;
    __syncthreads();
    if (c < 64) {
        float u[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) u[i] = s[c * 8 + i];
        vuis::sg_store8(a.o, a.o.pad + t, c * 8, u);
    }
    if (t == 0 && c == 0) *a.whole = a.T;
}

struct BFinalArgs {
    const float* x;     // [C / 4][T][4], activated
    const float* w;     // [C][7]
    const float* bias;  // [1]
    float* audio;       // [T]
    int T;
};

// Last convolution (C -> 1, k = 7) and the clamp: bound by reading x once.  A CTA takes 256 outputs; the 262 rows of four channels
// that they need are in shared memory twice over, the next four arrive while these are summed.
template <int C>
static __global__ void __launch_bounds__(256) k_bfinal(BFinalArgs a) {
    __shared__ __align__(16) float4 xs[2][262];
    __shared__ float ws[C * 7];
    vuis::sg_pdl_wait();
    vuis::sg_pdl_launch();
    const int tid = threadIdx.x, t0 = blockIdx.x * 256, t = t0 + tid;
    for (int i = tid; i < C * 7; i += 256) ws[i] = __ldg(a.w + i);
    auto load = [&](int c4, int i) {
        const int r = t0 - 6 + i;
        return r >= 0 && r < a.T ? __ldcg(reinterpret_cast<const float4*>(a.x) + (long long)c4 * a.T + r) : make_float4(0, 0, 0, 0);
    };
    float4 n0 = load(0, tid), n1 = tid < 6 ? load(0, 256 + tid) : n0;
    float acc = __ldg(a.bias);
    for (int c4 = 0; c4 < C / 4; ++c4) {
        float4* b = xs[c4 & 1];
        b[tid] = n0;
        if (tid < 6) b[256 + tid] = n1;
        __syncthreads();
        if (c4 + 1 < C / 4) {
            n0 = load(c4 + 1, tid);
            if (tid < 6) n1 = load(c4 + 1, 256 + tid);
        }
        const float* w = ws + c4 * 28;
#pragma unroll
        for (int j = 0; j < 7; ++j) {
            const float4 v = b[tid + j];
            acc += w[j] * v.x + w[7 + j] * v.y + w[14 + j] * v.z + w[21 + j] * v.w;
        }
    }
    if (t < a.T) a.audio[t] = fminf(1.f, fmaxf(-1.f, acc));
}

}  // namespace vuib_codec_batch
