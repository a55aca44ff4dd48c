// Codec encoder (24 kHz audio -> 16 codebook indices per 80 ms frame), fp32: the device work of the reference's
// QwenCodecEncoder.forward (src/vui/qwen_codec.py:385-390) as StreamingCodecEncoder drives it over a fixed 10 s
// buffer (671-805): causal convolution stack with ELU and strides 4, 5, 6, 8 (278-311), an 8-layer causal
// transformer over 25 Hz frames with LayerNorm, rotate-half RoPE, GELU MLP and per-channel layer scales (314-365),
// a stride-2 convolution to 12.5 Hz, and split residual vector quantisation: nearest code of 2048, residual
// subtracted, next codebook (185-275).
//
// Every convolution but the first and every linear layer is a split GEMM (split_gemm.cuh); its epilogues apply the ELU,
// GELU, layer scale and residual of what follows.  Here are the two ends: the one-channel input convolution and the quantiser.
#pragma once
#include "split_ops.cuh"

namespace vuie {

using vuis::SgPlanes;

struct EInArgs {
    const float* audio;  // [T]
    const float* w;      // [64][7]
    const float* bias;   // [64]
    float* y;            // [16][T][4]
    SgPlanes o;          // ELU(y)
    int T;
};

// CausalConv1d(1, 64, 7) (qwen_codec.py:278-311): 7 inputs per row, 10 bytes per channel out, so it is bound by its stores
// (64 channels of 240 000 rows: 154 MB).  A thread takes 32 channels of a row; rows of a warp are neighbours, so that every
// 16-byte store of a warp is a run of 512 bytes.
static __global__ void __launch_bounds__(256) k_ein(EInArgs a) {
    __shared__ float ws[64][8], bs[64];
    for (int i = threadIdx.x; i < 64 * 7; i += 256) ws[i / 7][i % 7] = a.w[i];
    if (threadIdx.x < 64) bs[threadIdx.x] = a.bias[threadIdx.x];
    vuis::sg_pdl_wait();
    vuis::sg_pdl_launch();
    __syncthreads();
    const int t = blockIdx.x * 128 + (threadIdx.x & 127), c0 = (threadIdx.x >> 7) * 32;
    float x[7];
#pragma unroll
    for (int j = 0; j < 7; ++j) x[j] = t - 6 + j >= 0 && t < a.T ? __ldg(a.audio + t - 6 + j) : 0.f;
#pragma unroll
    for (int i = 0; i < 32; i += 8) {
        float v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            float s = bs[c0 + i + q];
#pragma unroll
            for (int j = 0; j < 7; ++j) s += ws[c0 + i + q][j] * x[j];
            v[q] = s;
        }
        const int c = c0 + i;
        if (t < a.T) {
            *reinterpret_cast<float4*>(a.y + ((long long)(c / 4) * a.T + t) * 4) = make_float4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<float4*>(a.y + ((long long)(c / 4 + 1) * a.T + t) * 4) = make_float4(v[4], v[5], v[6], v[7]);
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = vuis::sg_act(v[q], vuis::SA_ELU, 0.f, 0.f);
            vuis::sg_store8(a.o, a.o.pad + t, c, v);
        }
        if (t < a.o.pad) {
            const float z[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            vuis::sg_store8(a.o, t, c, z);
        }
    }
}

// Residual vector quantisation (ResidualVQ.encode / EuclideanCodebook.encode, qwen_codec.py:190-195, 218-229): for each codebook
// the nearest of 2048 codes (first index on ties, as argmin), then the residual loses that code.  torch.cdist's distances are
// sqrt(|x|^2 + |e|^2 - 2 x.e) for inputs of this size; the argmin of |e|^2 - 2 x.e is the same.
struct ERvqArgs {
    const float* h;          // [512 / 4][T][4]: channels 0..255 projected for the semantic group, 256.. for the acoustic one
    const float* table[16];  // codebooks (2048, 256): 0 semantic, 1.. acoustic
    const float* norm2[16];  // |e|^2 per code (2048)
    long long* codes;        // [n_q][T]
    int n_q, T;
};

constexpr int RV_CL = 8, RV_F = 8;   // CTAs of a cluster, frames of a cluster

// A cluster of 8 CTAs takes 8 frames; CTA r compares them with codes [256 r, 256 r + 256) of each codebook in turn, so a codebook
// row read once serves 8 frames (one CTA a frame read all 2 MB of a codebook for each: 1.7 ms for 125 frames).  A lane holds 8
// of the 256 dimensions of all frames as pairs; per code 32 packed multiply-adds and 9 shuffles leave frame f's sum in the lanes
// with lane >> 2 == f.  The winners of the CTAs meet in every CTA's shared memory (two buffers in turn: the barrier of codebook
// i + 1 lies between the reads of i and the writes of i + 2).  grid (8 * ceil(T / 8), 2): semantic and acoustic groups side by side.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d)
        : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)), "l"(*reinterpret_cast<unsigned long long*>(&c)));
    return *reinterpret_cast<float2*>(&d);
}

constexpr int RV_WARPS = 16;

static __global__ void __cluster_dims__(RV_CL, 1, 1) __launch_bounds__(32 * RV_WARPS) k_ervq(ERvqArgs a) {
    __shared__ float wv[RV_WARPS][RV_F];
    __shared__ int wi[RV_WARPS][RV_F], pick[RV_F];
    __shared__ float cv[2][RV_CL][RV_F];
    __shared__ int ci[2][RV_CL][RV_F];
    constexpr int PER = 256 / RV_WARPS;
    const int part = blockIdx.y, n = part ? a.n_q - 1 : 1, q0 = part ? 1 : 0;
    if (n == 0) return;   // the whole cluster
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, f0 = (blockIdx.x / RV_CL) * RV_F, rank = blockIdx.x % RV_CL;
    // A peer's shared memory may be touched only once all CTAs of the cluster run: waited for in front of the first store to one.
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    vuis::sg_pdl_wait();
    vuis::sg_pdl_launch();
    float2 r[RV_F][4];
#pragma unroll
    for (int f = 0; f < RV_F; ++f) {
        const int t = min(f0 + f, a.T - 1);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float4 v = __ldcg(reinterpret_cast<const float4*>(a.h + ((long long)(part * 64 + lane * 2 + h) * a.T + t) * 4));
            r[f][2 * h] = make_float2(v.x, v.y);
            r[f][2 * h + 1] = make_float2(v.z, v.w);
        }
    }
    for (int cb = 0; cb < n; ++cb) {
        const float* E = a.table[q0 + cb];
        const float* N2 = a.norm2[q0 + cb];
        float bv = INFINITY;
        int bi = 0;
        const int first = rank * 256 + warp * PER;
        const float n2 = __ldg(N2 + first + lane % PER);
#pragma unroll 4
        for (int i = 0; i < PER; ++i) {
            const int c = first + i;
            const float4 e0 = __ldg(reinterpret_cast<const float4*>(E + (long long)c * 256 + lane * 8));
            const float4 e1 = __ldg(reinterpret_cast<const float4*>(E + (long long)c * 256 + lane * 8 + 4));
            const float2 e[4] = {make_float2(e0.x, e0.y), make_float2(e0.z, e0.w), make_float2(e1.x, e1.y), make_float2(e1.z, e1.w)};
            float d[RV_F];
#pragma unroll
            for (int f = 0; f < RV_F; ++f) {
                float2 s2 = make_float2(0.f, 0.f);
#pragma unroll
                for (int q = 0; q < 4; ++q) s2 = fma2(r[f][q], e[q], s2);
                d[f] = s2.x + s2.y;
            }
            const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
            float d4[4], d2[2];
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                const float keep = b4 ? d[f + 4] : d[f], give = b4 ? d[f] : d[f + 4];
                d4[f] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
            }
#pragma unroll
            for (int f = 0; f < 2; ++f) {
                const float keep = b3 ? d4[f + 2] : d4[f], give = b3 ? d4[f] : d4[f + 2];
                d2[f] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
            }
            float s = (b2 ? d2[1] : d2[0]) + __shfl_xor_sync(0xffffffffu, b2 ? d2[0] : d2[1], 4);
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            const float dist = __shfl_sync(0xffffffffu, n2, i) - 2.f * s;
            if (dist < bv) { bv = dist; bi = c; }    // c ascends: the first minimum is kept
        }
        if ((lane & 3) == 0) { wv[warp][lane >> 2] = bv; wi[warp][lane >> 2] = bi; }
        __syncthreads();
        if (cb == 0) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        const int buf = cb & 1;
        if (tid < RV_CL * RV_F) {
            const int f = tid & 7, dst = tid >> 3;
            float v = wv[0][f];
            int w = wi[0][f];
            for (int i = 1; i < RV_WARPS; ++i)
                if (wv[i][f] < v) { v = wv[i][f]; w = wi[i][f]; }
            const uint32_t av = vuis::sg_smem(&cv[buf][rank][f]), ai = vuis::sg_smem(&ci[buf][rank][f]);
            asm volatile("{\n\t.reg .b32 ra, rb;\n\tmapa.shared::cluster.u32 ra, %0, %2;\n\tmapa.shared::cluster.u32 rb, %1, %2;\n\t"
                         "st.shared::cluster.f32 [ra], %3;\n\tst.shared::cluster.s32 [rb], %4;\n\t}"
                         ::"r"(av), "r"(ai), "r"(dst), "f"(v), "r"(w) : "memory");
        }
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (tid < RV_F) {
            float v = cv[buf][0][tid];
            int w = ci[buf][0][tid];
            for (int i = 1; i < RV_CL; ++i)
                if (cv[buf][i][tid] < v) { v = cv[buf][i][tid]; w = ci[buf][i][tid]; }
            pick[tid] = w;
            if (rank == 0 && f0 + tid < a.T) a.codes[(long long)(q0 + cb) * a.T + f0 + tid] = w;
        }
        __syncthreads();
#pragma unroll
        for (int f = 0; f < RV_F; ++f) {
            const float* e = E + (long long)pick[f] * 256 + lane * 8;
            const float4 e0 = __ldg(reinterpret_cast<const float4*>(e)), e1 = __ldg(reinterpret_cast<const float4*>(e + 4));
            r[f][0].x -= e0.x; r[f][0].y -= e0.y; r[f][1].x -= e0.z; r[f][1].y -= e0.w;
            r[f][2].x -= e1.x; r[f][2].y -= e1.y; r[f][3].x -= e1.z; r[f][3].y -= e1.w;
        }
    }
}

}  // namespace vuie
