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
    int* flag;
};

constexpr int RV_CL = 8;                   // CTAs of a cluster
constexpr int RV_RESIDENT = 15;   // clusters of 8 CTAs with this much shared memory that run at once
constexpr int RV_WARPS = 16, RV_CODES = 4, RV_STAGES = 3;   // a ring stage: four codes (4 KB) of one warp
constexpr int RV_SMEM = RV_WARPS * RV_STAGES * RV_CODES * 1024;

// A cluster of 8 CTAs takes F frames; CTA r compares them with codes [256 r, 256 r + 256) of each codebook in turn, so a codebook
// row read once serves F frames (one CTA a frame read all 2 MB of a codebook for each: 1.7 ms for 125 frames).  The codebooks are a
// chain, 15 times over: distances, exchange of the winners, the winners' rows.  What bounds a link is instructions and round trips:
//  * The codes do not depend on the residual, so every warp streams its 16 of a codebook through a ring of its own (bulk copies; three
//    quarters of the next codebook's are there before the exchange is over).
//  * A lane holds 8 of the 256 dimensions of all frames as pairs; per code 32 packed multiply-adds and 9 shuffles leave frame f's sum in
//    the lanes with lane >> 2 == f (a ninth frame: 5 more, in every lane).  With eight lanes a code and two frames a lane there are 3
//    shuffles, but each 16-byte load is four passes of shared memory however many lanes share it: 8.4 us a codebook.
//  * The winners of the CTAs are pushed into every CTA's shared memory and counted there (one hop; two buffers and two barriers in
//    turn: a CTA pushes for codebook i + 2 only once it has this one's push for i + 1, which comes after i was read).
// grid (8 * ceil(T / F), 2): acoustic codebooks first, the semantic one beside.  F is 9 where that takes a wave of resident clusters less
// than 8 (121 to 135 frames, the 10 s buffer among them; 241 to 250: an encode of 250 frames 2.23 -> 2.20 ms).
// 13 frames 107 us (140 with loads in the loop and a cluster barrier a codebook), 80 frames 114 (137), 125 frames 156 (266).
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d)
        : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)), "l"(*reinterpret_cast<unsigned long long*>(&c)));
    return *reinterpret_cast<float2*>(&d);
}

// (distance, code) as a number whose order is that of the distances, the lower code first among equals.
__device__ __forceinline__ unsigned long long rv_key(float v, int i) {
    const unsigned b = __float_as_uint(v);
    return (unsigned long long)((b & 0x80000000u) ? ~b : (b | 0x80000000u)) << 32 | (unsigned)i;
}

template <int F>
static __global__ void __cluster_dims__(RV_CL, 1, 1) __launch_bounds__(32 * RV_WARPS) k_ervq(ERvqArgs a) {
    static_assert(F == 8 || F == 9, "eight frames by halves, a ninth by itself");
    extern __shared__ __align__(128) unsigned char rv_ring[];   // [warp][stage][code][256]
    // This CTA's best of each warp, two buffers in turn: a warp that has the peers' answers writes codebook i + 1's while a thread that answers
    // another CTA may still be reading i's; that thread passes the barrier of i + 1 before anything of i + 2 is written.
    __shared__ unsigned long long won[2][RV_WARPS][F];
    __shared__ __align__(8) unsigned long long peers[2][RV_CL][F];
    __shared__ uint64_t full[RV_WARPS][RV_STAGES], got[2];
    constexpr int PER = 256 / RV_WARPS, LOADS = PER / RV_CODES;
    const int part = 1 - blockIdx.y, n = part ? a.n_q - 1 : 1, q0 = part ? 1 : 0;
    if (n == 0) return;   // the whole cluster
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, f0 = (blockIdx.x / RV_CL) * F, rank = blockIdx.x % RV_CL;
    if (tid == 0) {
        for (int w = 0; w < RV_WARPS; ++w)
            for (int i = 0; i < RV_STAGES; ++i) vuis::sg_bar_init(&full[w][i], 1);
        for (int i = 0; i < 2; ++i) vuis::sg_bar_init(&got[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        for (int i = 0; i < 2; ++i) vuis::sg_bar_expect(&got[i], RV_CL * F * 8);
    }
    __syncthreads();
    // A peer's shared memory may be touched only once all CTAs of the cluster run: waited for in front of the first store to one.
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    const int first = rank * 256 + warp * PER;
    unsigned char* const ring = rv_ring + warp * (RV_STAGES * RV_CODES * 1024);
    auto request = [&](int load) {   // this warp's load-th stage over all codebooks (one lane)
        const int cb = load / LOADS, st = load % RV_STAGES;
        vuis::sg_bar_expect(&full[warp][st], RV_CODES * 1024);
        vuis::sg_bulk(ring + st * RV_CODES * 1024, a.table[q0 + cb] + (size_t)(first + (load % LOADS) * RV_CODES) * 256, RV_CODES * 1024, &full[warp][st]);
    };
    if (lane == 0)
        for (int i = 0; i < RV_STAGES; ++i) request(i);   // a codebook is more stages than the ring
    __syncwarp();
    float n2 = __ldg(a.norm2[q0] + first + lane % PER);
    vuis::sg_pdl_wait();
    vuis::sg_pdl_launch();
    bool bad = false;
    unsigned limit = vuis::SG_SPIN_LIMIT;
    float2 r[F][4];   // dims 4 lane .. + 3 and 128 + 4 lane .. + 3
#pragma unroll
    for (int f = 0; f < F; ++f) {
        const int t = min(f0 + f, a.T - 1);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float4 v = __ldcg(reinterpret_cast<const float4*>(a.h + ((long long)(part * 64 + h * 32 + lane) * a.T + t) * 4));
            r[f][2 * h] = make_float2(v.x, v.y);
            r[f][2 * h + 1] = make_float2(v.z, v.w);
        }
    }
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
    const int loads = n * LOADS;
    for (int cb = 0, load = 0; cb < n; ++cb) {
        float bv = INFINITY, bv8 = INFINITY;
        int bi = 0, bi8 = 0;
        for (int k = 0; k < LOADS; ++k, ++load) {
            const int st = load % RV_STAGES;
            if (!vuis::sg_bar_wait(&full[warp][st], (load / RV_STAGES) & 1, limit)) { bad = true; limit = 16; }
            const float4* e = reinterpret_cast<const float4*>(ring + st * RV_CODES * 1024) + lane;
            float4 ev[RV_CODES][2];
#pragma unroll
            for (int c = 0; c < RV_CODES; ++c) { ev[c][0] = e[c * 64]; ev[c][1] = e[c * 64 + 32]; }
#pragma unroll
            for (int c = 0; c < RV_CODES; ++c) {
                const float2 v[4] = {make_float2(ev[c][0].x, ev[c][0].y), make_float2(ev[c][0].z, ev[c][0].w), make_float2(ev[c][1].x, ev[c][1].y),
                                     make_float2(ev[c][1].z, ev[c][1].w)};
                float d[F];
#pragma unroll
                for (int f = 0; f < F; ++f) {
                    float2 s2 = make_float2(0.f, 0.f);
#pragma unroll
                    for (int q = 0; q < 4; ++q) s2 = fma2(r[f][q], v[q], s2);
                    d[f] = s2.x + s2.y;
                }
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
                const float e2 = __shfl_sync(0xffffffffu, n2, k * RV_CODES + c);
                const int code = first + k * RV_CODES + c;
                const float dist = e2 - 2.f * s;
                if (dist < bv) { bv = dist; bi = code; }    // codes ascend: the first minimum is kept
                if constexpr (F == 9) {
#pragma unroll
                    for (int x = 16; x > 0; x >>= 1) d[8] += __shfl_xor_sync(0xffffffffu, d[8], x);
                    const float dist8 = e2 - 2.f * d[8];
                    if (dist8 < bv8) { bv8 = dist8; bi8 = code; }
                }
            }
            __syncwarp();
            if (lane == 0 && load + RV_STAGES < loads) request(load + RV_STAGES);
        }
        if (cb + 1 < n) n2 = __ldg(a.norm2[q0 + cb + 1] + first + lane % PER);
        const int buf = cb & 1;
        if ((lane & 3) == 0) won[buf][warp][lane >> 2] = rv_key(bv, bi);
        if (F == 9 && lane == 0) won[buf][warp][8] = rv_key(bv8, bi8);
        __syncthreads();
        if (cb == 0) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (tid < RV_CL * F) {
            const int f = tid % F, dst = tid / F;
            unsigned long long w[RV_WARPS];
#pragma unroll
            for (int i = 0; i < RV_WARPS; ++i) w[i] = won[buf][i][f];
#pragma unroll
            for (int k = RV_WARPS / 2; k > 0; k /= 2)
#pragma unroll
                for (int i = 0; i < k; ++i) w[i] = min(w[i], w[i + k]);
            asm volatile("{\n\t.reg .b32 ra, rb;\n\tmapa.shared::cluster.u32 ra, %0, %2;\n\tmapa.shared::cluster.u32 rb, %1, %2;\n\t"
                         "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [ra], %3, [rb];\n\t}"
                         ::"r"(vuis::sg_smem(&peers[buf][rank][f])), "r"(vuis::sg_smem(&got[buf])), "r"(dst), "l"(w[0]) : "memory");
        }
        {
            const uint32_t bar = vuis::sg_smem(&got[buf]);
            uint32_t ok = 0;
            for (unsigned i = 0; i < limit && !ok; ++i)
                asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                             : "=r"(ok) : "r"(bar), "r"((unsigned)(cb >> 1) & 1) : "memory");
            if (!ok) { bad = true; limit = 16; }
        }
        // lane: CTA lane & 7's answers for frames lane >> 3, lane >> 3 + 4 and 8
        int pick[F];
        {
            unsigned long long p[3];
#pragma unroll
            for (int i = 0; i < (F == 9 ? 3 : 2); ++i) {
                p[i] = peers[buf][lane & 7][i == 2 ? 8 : (lane >> 3) + 4 * i];
#pragma unroll
                for (int x = 4; x > 0; x >>= 1) p[i] = min(p[i], __shfl_xor_sync(0xffffffffu, p[i], x));
            }
#pragma unroll
            for (int f = 0; f < F; ++f)   // an index also where the wait ran out
                pick[f] = __shfl_sync(0xffffffffu, (int)p[f >> 2], f == 8 ? 0 : (f & 3) * 8) & 2047;
        }
        if (rank == 0 && warp == 0) {
#pragma unroll
            for (int f = 0; f < F; ++f)
                if (lane == f && f0 + f < a.T) a.codes[(long long)(q0 + cb) * a.T + f0 + f] = pick[f];
        }
        if (cb + 1 == n) break;
#pragma unroll
        for (int f = 0; f < F; ++f) {
            const float4* e = reinterpret_cast<const float4*>(a.table[q0 + cb] + (size_t)pick[f] * 256) + lane;
            const float4 e0 = __ldg(e), e1 = __ldg(e + 32);
            r[f][0].x -= e0.x; r[f][0].y -= e0.y; r[f][1].x -= e0.z; r[f][1].y -= e0.w;
            r[f][2].x -= e1.x; r[f][2].y -= e1.y; r[f][3].x -= e1.z; r[f][3].y -= e1.w;
        }
        // armed for codebook cb + 2, whose first push follows this CTA's next one (behind the barrier above)
        if (tid == 0) vuis::sg_bar_expect(&got[buf], RV_CL * F * 8);
    }
    if (bad) {   // what may still be on its way to this CTA's shared memory lands before the CTA retires
        if (lane == 0) atomicOr(a.flag, vuis::SG_FLAG_WAIT);
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    }
    __syncthreads();
}

}  // namespace vuie
