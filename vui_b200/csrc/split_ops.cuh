// Row-wise kernels between the split GEMMs (split_gemm.cuh): normalisation and causal attention in fp32.  They read fp32
// activations [C / 4][T][4] as a GEMM's epilogue leaves them and write the next GEMM's planes.
#pragma once
#include "split_gemm.cuh"

namespace vuis {

enum { SN_RMS = 0, SN_LAYER = 1, SN_DW_LAYER = 2 };

struct SNormArgs {
    const float* x;        // [C / 4][x_rows][4]
    int x_rows;
    const float* w;        // [C]
    const float* b;        // [C] (SN_LAYER, SN_DW_LAYER)
    const float* dw_w;     // [C][7] depthwise weights (SN_DW_LAYER: causal convolution over time first)
    const float* dw_b;     // [C]
    float eps;
    SgPlanes o;
    int T;
};

// Norm over C channels of every row.  A CTA takes 8 rows: thread (row r, group g of 32) holds the eight-channel chunks g, g + 32, ...
// in registers, so x is read once and mean and variance are two exact passes; 16 to 64 CTAs of latency-bound work.
template <int MODE, int C>
__global__ void __launch_bounds__(256) k_snorm(SNormArgs a) {
    constexpr int NV = C / 256;
    __shared__ float red[2][8][8];
    sg_pdl_wait();
    sg_pdl_launch();
    const int r = threadIdx.x & 7, g = threadIdx.x >> 3, warp = threadIdx.x >> 5, t = blockIdx.x * 8 + r;
    float v[NV][8];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int c = (g + 32 * i) * 8;
        if (MODE != SN_DW_LAYER) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float4 q = t < a.T ? __ldcg(reinterpret_cast<const float4*>(a.x + ((long long)(c / 4 + h) * a.x_rows + t) * 4)) : make_float4(0, 0, 0, 0);
                v[i][4 * h] = q.x; v[i][4 * h + 1] = q.y; v[i][4 * h + 2] = q.z; v[i][4 * h + 3] = q.w;
            }
        } else {
#pragma unroll
            for (int q = 0; q < 8; ++q) v[i][q] = __ldg(a.dw_b + c + q);
#pragma unroll
            for (int j = 0; j < 7; ++j) {
                const int tj = t - 6 + j;
                const bool on = tj >= 0 && t < a.T;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float4 q = on ? __ldcg(reinterpret_cast<const float4*>(a.x + ((long long)(c / 4 + h) * a.x_rows + tj) * 4)) : make_float4(0, 0, 0, 0);
                    const float* dw = a.dw_w + (c + 4 * h) * 7 + j;
                    v[i][4 * h] += __ldg(dw) * q.x; v[i][4 * h + 1] += __ldg(dw + 7) * q.y;
                    v[i][4 * h + 2] += __ldg(dw + 14) * q.z; v[i][4 * h + 3] += __ldg(dw + 21) * q.w;
                }
            }
        }
    }
    // sums over the channels of a row: lanes r, r + 8, r + 16, r + 24 of every warp hold it
    auto row_sum = [&](float s, int which) {
        s += __shfl_xor_sync(0xffffffffu, s, 8);
        s += __shfl_xor_sync(0xffffffffu, s, 16);
        if ((threadIdx.x & 31) < 8) red[which][warp][r] = s;
        __syncthreads();
        float sum = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) sum += red[which][w][r];
        return sum;
    };
    float mean = 0.f, s = 0.f;
    if (MODE != SN_RMS) {
#pragma unroll
        for (int i = 0; i < NV; ++i)
#pragma unroll
            for (int q = 0; q < 8; ++q) s += v[i][q];
        mean = row_sum(s, 0) / (float)C;
        s = 0.f;
    }
#pragma unroll
    for (int i = 0; i < NV; ++i)
#pragma unroll
        for (int q = 0; q < 8; ++q) { const float d = v[i][q] - mean; s += d * d; }
    const float rinv = rsqrtf(row_sum(s, 1) / (float)C + a.eps);
    if (t >= a.T) return;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int c = (g + 32 * i) * 8;
        float o[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) o[q] = (v[i][q] - mean) * rinv * __ldg(a.w + c + q) + (MODE == SN_RMS ? 0.f : __ldg(a.b + c + q));
        sg_store8(a.o, a.o.pad + t, c, o);
    }
}

struct SAttnArgs {
    const float* qkv;      // q | k | v, H * 64 channels each: [3 * H * 16][rows][4], before RoPE
    int rows;
    const float* rope;     // [8][rope_rows][8]: cos, sin of channels 4 i .. 4 i + 3 (the same for the other half of a head), k_srope
    int rope_rows;
    SgPlanes o;            // H * 64 channels
    int T, H;
    int cluster;           // sat_cluster(T)
};

// Rotate-half tables [T][64] (both halves alike) in the order in which k_sattn's lanes, one a row, read them.
static __global__ void __launch_bounds__(256) k_srope(const float* cos_t, const float* sin_t, float* out, int T) {
    const int i = blockIdx.x * 256 + threadIdx.x, t = i / 32, d = i % 32;
    if (t >= T) return;
    float* o = out + ((long long)(d / 4) * T + t) * 8 + d % 4;
    o[0] = cos_t[t * 64 + d];
    o[4] = sin_t[t * 64 + d];
}

constexpr int SAT_Q = 16, SAT_K = 64;   // queries of a CTA, keys of a step

// Causal attention with rotate-half RoPE, head size 64: a CTA takes 16 queries of a head (two a warp), keys arrive 64 at a time in
// shared memory (RoPE applied on the way), softmax with a running maximum per step.  T <= 500, so there are a few hundred CTAs of
// work that is a chain of loads, two products and a softmax, 5 us a step: the steps of 16 queries are shared out over a cluster of up
// to SAT_CL CTAs, whose states the first one merges in their order (rows 250 / 160 / 96: 13.7 / 9.4 / 8.9 us a layer, 24.7 / 16.9 / 10.6
// with all steps in one CTA).
// Every load is a row per lane (with the tables as [T][64] a lane fetched a line of its own: 35 us a layer of 250 rows); a CTA's next
// step, where it has one, is requested before this one's products.
constexpr int SAT_CL = 4;
inline int sat_cluster(int T) { return T <= SAT_K ? 1 : T <= 2 * SAT_K ? 2 : SAT_CL; }

template <int PER_SM>
static __global__ void __launch_bounds__(256, PER_SM) k_sattn(SAttnArgs a) {
    __shared__ __align__(16) float qs[SAT_Q][64], ks[SAT_K][65], vs[SAT_K][64], ps[8][2][SAT_K];
    static_assert(sizeof(vs) >= SAT_Q * 66 * sizeof(float), "a CTA's o[64], m, l of every query take the place of its values");
    const int CL = a.cluster, rank = blockIdx.x % CL;
    sg_pdl_wait();
    sg_pdl_launch();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h = blockIdx.y, q0 = blockIdx.x / CL * SAT_Q, T = a.T;
    const int last = min(q0 + SAT_Q, T), own = rank * SAT_K, step = CL * SAT_K;   // keys [0, last); this CTA's first, and from step to step
    if (own >= last) return;   // nothing to add, and nobody looks here
    const float* xq = a.qkv + (long long)h * 16 * a.rows * 4;
    const float* xk = xq + (long long)a.H * 16 * a.rows * 4;
    const float* xv = xk + (long long)a.H * 16 * a.rows * 4;
    auto row4 = [&](const float* x, int c4, int t) { return __ldcg(reinterpret_cast<const float4*>(x + ((long long)c4 * a.rows + t) * 4)); };
    auto table = [&](int i, int t, int w) { return __ldg(reinterpret_cast<const float4*>(a.rope + ((long long)i * a.rope_rows + t) * 8 + w)); };
    // rotate-half: channel d pairs with d + 32; an item is four channels of both halves of one row
    auto rotate = [](float4 u, float4 w, float4 c, float4 s, float (&lo)[4], float (&hi)[4]) {
        lo[0] = u.x * c.x - w.x * s.x; lo[1] = u.y * c.y - w.y * s.y; lo[2] = u.z * c.z - w.z * s.z; lo[3] = u.w * c.w - w.w * s.w;
        hi[0] = w.x * c.x + u.x * s.x; hi[1] = w.y * c.y + u.y * s.y; hi[2] = w.z * c.z + u.z * s.z; hi[3] = w.w * c.w + u.w * s.w;
    };
    float4 f[2][6];   // two items of the next step: K halves, V halves, cos, sin
    auto fetch = [&](int k0) {
#pragma unroll
        for (int it = 0; it < 2; ++it) {
            const int i = (tid >> 6) + 4 * it, t = min(k0 + (tid & 63), T - 1);
            f[it][0] = row4(xk, i, t); f[it][1] = row4(xk, i + 8, t);
            f[it][2] = row4(xv, i, t); f[it][3] = row4(xv, i + 8, t);
            f[it][4] = table(i, t, 0); f[it][5] = table(i, t, 4);
        }
    };
    fetch(own);
    if (tid < 128) {
        const int q = tid & 15, i = tid >> 4, t = min(q0 + q, T - 1);
        float lo[4], hi[4];
        rotate(row4(xq, i, t), row4(xq, i + 8, t), table(i, t, 0), table(i, t, 4), lo, hi);
#pragma unroll
        for (int d = 0; d < 4; ++d) { qs[q][4 * i + d] = lo[d] * 0.125f; qs[q][4 * i + 32 + d] = hi[d] * 0.125f; }
    }
    float m[2], l[2], o[2][2];
#pragma unroll
    for (int i = 0; i < 2; ++i) { m[i] = -INFINITY; l[i] = 0.f; o[i][0] = o[i][1] = 0.f; }
    for (int k0 = own; k0 < last; k0 += step) {
        __syncthreads();
#pragma unroll
        for (int it = 0; it < 2; ++it) {
            const int k = tid & 63, d = ((tid >> 6) + 4 * it) * 4;
            float lo[4], hi[4];
            rotate(f[it][0], f[it][1], f[it][4], f[it][5], lo, hi);
#pragma unroll
            for (int q = 0; q < 4; ++q) { ks[k][d + q] = lo[q]; ks[k][d + 32 + q] = hi[q]; }
            *reinterpret_cast<float4*>(&vs[k][d]) = f[it][2];
            *reinterpret_cast<float4*>(&vs[k][d + 32]) = f[it][3];
        }
        __syncthreads();
        if (k0 + step < last) fetch(k0 + step);
        float s[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll 4
        for (int d = 0; d < 64; d += 4) {
            float kv[2][4];
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int q = 0; q < 4; ++q) kv[u][q] = ks[lane + 32 * u][d + q];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float4 qv = *reinterpret_cast<const float4*>(&qs[warp * 2 + i][d]);
#pragma unroll
                for (int u = 0; u < 2; ++u) s[i][u] += qv.x * kv[u][0] + qv.y * kv[u][1] + qv.z * kv[u][2] + qv.w * kv[u][3];
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int t = q0 + warp * 2 + i;
            if (k0 + lane > t) s[i][0] = -INFINITY;
            if (k0 + lane + 32 > t) s[i][1] = -INFINITY;
            float mx = fmaxf(s[i][0], s[i][1]);
#pragma unroll
            for (int w = 16; w > 0; w >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, w));
            const float mn = fmaxf(m[i], mx);
            // a query before all keys of the step (not of the first CTA's first one) has no state yet
            const float ref = mn == -INFINITY ? 0.f : mn;
            const float corr = expf(m[i] - ref), p0 = expf(s[i][0] - ref), p1 = expf(s[i][1] - ref);
            ps[warp][i][lane] = p0;
            ps[warp][i][lane + 32] = p1;
            float sum = p0 + p1;
#pragma unroll
            for (int w = 16; w > 0; w >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, w);
            l[i] = l[i] * corr + sum;
            o[i][0] *= corr;
            o[i][1] *= corr;
            m[i] = mn;
        }
        __syncwarp();
#pragma unroll 4
        for (int k = 0; k < SAT_K; k += 4) {
            float4 p[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) p[i] = *reinterpret_cast<const float4*>(&ps[warp][i][k]);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float v0 = vs[k + q][lane], v1 = vs[k + q][lane + 32];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const float pv = q == 0 ? p[i].x : q == 1 ? p[i].y : q == 2 ? p[i].z : p[i].w;
                    o[i][0] += pv * v0;
                    o[i][1] += pv * v1;
                }
            }
        }
    }
    if (CL > 1) {
        float* const mine = &vs[0][0];
        if (rank > 0) {
            __syncthreads();
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                float* p = mine + (warp * 2 + i) * 66;
                p[lane] = o[i][0];
                p[lane + 32] = o[i][1];
                if (lane == 0) { p[64] = m[i]; p[65] = l[i]; }
            }
        }
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (rank == 0) {
            float v[SAT_CL - 1][2][4];   // all requested before the first is used
#pragma unroll
            for (int r = 1; r < SAT_CL; ++r)
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    if (r < CL && r * SAT_K < last) {
                        uint32_t src;
                        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(src) : "r"(sg_smem(mine + (warp * 2 + i) * 66)), "r"(r));
                        asm volatile("ld.shared::cluster.f32 %0, [%4];\n\tld.shared::cluster.f32 %1, [%4 + 128];\n\tld.shared::cluster.f32 %2, [%5 + 256];\n\t"
                                     "ld.shared::cluster.f32 %3, [%5 + 260];"
                                     : "=&f"(v[r - 1][i][0]), "=&f"(v[r - 1][i][1]), "=&f"(v[r - 1][i][2]), "=&f"(v[r - 1][i][3])
                                     : "r"(src + lane * 4), "r"(src) : "memory");
                    }
#pragma unroll
            for (int r = 1; r < SAT_CL; ++r)
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    if (r < CL && r * SAT_K < last) {   // key 0 is in this CTA, so m is finite
                        const float mn = fmaxf(m[i], v[r - 1][i][2]), c0 = expf(m[i] - mn), c1 = expf(v[r - 1][i][2] - mn);
                        l[i] = l[i] * c0 + v[r - 1][i][3] * c1;
                        o[i][0] = o[i][0] * c0 + v[r - 1][i][0] * c1;
                        o[i][1] = o[i][1] * c0 + v[r - 1][i][1] * c1;
                        m[i] = mn;
                    }
        }
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");   // read before its CTA retires
        if (rank > 0) return;
    }
    // through shared memory to eight-channel chunks (a warp's rows of qs are its own)
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        qs[warp * 2 + i][lane] = o[i][0] / l[i];
        qs[warp * 2 + i][lane + 32] = o[i][1] / l[i];
    }
    __syncwarp();
    const int q = warp * 2 + (lane >> 3 & 1), c = (lane & 7) * 8;
    if (lane < 16 && q0 + q < T) {
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = qs[q][c + i];
        sg_store8(a.o, a.o.pad + q0 + q, h * 64 + c, v);
    }
}

inline cudaError_t sat_launch(const SgCtx& x, SAttnArgs a) {
    a.cluster = sat_cluster(a.T);
    const dim3 grid((a.T + SAT_Q - 1) / SAT_Q * a.cluster, a.H);
    if (a.cluster == 1) return sg_run(x, k_sattn<2>, grid, dim3(256), 0, a);
    // CTAs with keys to look at; where two to an SM (128 registers) are a wave and a bit, three (80): 250 rows of eight heads 13.7 us, not
    // 17.0, but 160 rows 12.7, not 9.4
    int busy = 0;
    for (int q0 = 0; q0 < a.T; q0 += SAT_Q) {
        const int last = q0 + SAT_Q < a.T ? q0 + SAT_Q : a.T, steps = (last + SAT_K - 1) / SAT_K;
        busy += steps < a.cluster ? steps : a.cluster;
    }
    return sg_run_cluster(x, busy * a.H > 2 * x.num_sms ? k_sattn<3> : k_sattn<2>, a.cluster, grid, dim3(256), 0, a);
}

}  // namespace vuis
