// fp32 convolutions and linear layers on the 5th-generation tensor cores, without giving up fp32 accuracy: every operand is
// the sum of three bf16 planes (hi + mid + lo, 8 mantissa bits each: all 24 of an fp32 value), and a product is the six plane
// products that lie above 2^-24 of it (hi hi | hi mid, mid hi, mid mid, hi lo, lo hi).
//
//   D[t][n] = sum_{tap, c} X[t + (tap - (taps - 1)) * dil][c] * W[tap][n][c]          (causal convolution; taps = 1: a matrix)
//
// is one GEMM: t is the MMA's M side (128 rows a tile), n its N side (NT = 32, 64, 96 or 128 columns), and the taps share the
// input rows that are already in shared memory.
//
//  * Activations are stored as planes [3][C / 32][rows][32] bf16 whose 64-byte rows already lie in the 64-byte-swizzled order
//    of the MMA's operand tiles.  A window of rows of one 32-channel group is therefore ONE contiguous run per plane (a
//    cp.async.bulk each, no tensor map), and a tap is the same window read from a start address `dil` rows further down: the
//    swizzle is a function of address bits, so a shifted start needs no copy.  `pad` zero rows in front are the causal padding.
//  * A convolution of stride s and kernel 2 s is a 2-tap convolution over s * C channels: its producer stores row t of phase
//    t mod s at row t / s of channel group (t mod s) * C / 32 + ... (SgOut::p_div).  A transposed convolution of stride s and
//    kernel 2 s is a 2-tap convolution with s * Cout columns, whose column (j, co) is written to row t * s + j (SgOut::up).
//  * Weights are packed once, per (column tile, 32-channel group, tap), as the 3 x NT x 64-byte image of a ring stage: one
//    contiguous bulk copy a stage.
//  * Two accumulators in tensor memory: hi * hi, and the sum of the five small products.  The tensor cores round the running
//    sum towards zero, so a long chain would drift; apart, the small products are not cut off by the large sum, and after
//    every SG_SEG chunks the pair is read out and added to fp32 registers (round to nearest).  A second pair lets the MMAs of
//    the next segment or tile go on meanwhile.
//  * A_hi * [B_hi | B_mid] is one MMA of 2 NT columns that fills both accumulators (the planes lie behind one another): five
//    instructions per 16 channels, and the A tile is read once less from shared memory, whose port is what bounds NT < 128.
//
// Warps: 0 input windows, 1 weights (both bulk copies, mbarrier rings), 2 MMAs (one elected lane), 4..11 epilogue.  The grid is
// persistent: one CTA per SM walks the tiles, column tiles of the same rows next to one another, so that they share L2 lines.
// Every wait is bounded (SgArgs::spin_limit) and leaves SG_FLAG_WAIT; after the first that runs out the others give up at once.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace vuis {

typedef __nv_bfloat16 bf16;

constexpr int SG_THREADS = 384, SG_EPI_WARPS = 8;
constexpr int SG_M = 128;            // rows of a tile
constexpr int SG_MAX_A = 8, SG_MAX_B = 12;
constexpr int SG_PAD = 64;           // most zero rows in front of an input (history of a k = 7, dilation 9 convolution is 54)
constexpr int SG_SMEM = 212 * 1024;
constexpr int SG_FLAG_WAIT = 4;
constexpr unsigned SG_SPIN_LIMIT = 1u << 22;

enum { SA_NONE = 0, SA_SNAKE = 1, SA_ELU = 2, SA_GELU = 3 };

// Planes of an activation: element (plane, row, channel) of [3][groups][rows][32], see sg_plane_offset.
struct SgPlanes {
    bf16* p;
    long long plane, group;   // elements between planes, between 32-channel groups
    int pad;                  // row of time 0
};

struct SgOut {
    const float* bias;    // [Cout] or null
    const float* scale;   // [Cout] or null: v = res + scale * v
    const float* res;     // like y, or null
    float* y;             // fp32 [Cout / 4][y_rows][4] or null
    int y_rows;
    int y_act;            // y gets act(v) instead of v
    SgPlanes o;           // planes of act(v), or o.p null
    int p_div;            // row t goes to phase t % p_div, row t / p_div (the input order of a strided convolution)
    int act;              // SA_*
    const float* ea;      // SnakeBeta parameters [Cout]
    const float* ib;
    int Cout;             // channels; columns are (j, co) of a transposed convolution of stride `up`, (gate, up) pairs if gated
    int up;
    int gated;            // columns 2 i, 2 i + 1 -> channel i = silu(v[2 i]) * v[2 i + 1]
};

struct SgArgs {
    SgPlanes x;
    const bf16* w;        // packed weights
    int kchunks;          // 32-channel groups of the input
    int dil;
    int M, n_tiles, m_tiles;
    int b_keep;           // a CTA's tiles share one column tile whose weights fit the ring: they are fetched once
    int splits;           // CTAs of a cluster that share a tile's channels: 1, 2, 4 or 8
    SgOut out;
    int* flag;
    unsigned spin_limit;
};

// Ring of a kernel: G groups of `TAPS` weight stages, GA windows (as many as 211 KB hold; a round trip from a freed stage to its
// next contents takes about 1500 cycles, a chunk of NT = 32 about 416), and channel groups (of 32) between two read-outs of the
// accumulators: 4 to 7 chunks, 128 to 224 products.
template <int NT, int TAPS>
struct SgRing {
    static constexpr int G = TAPS == 7 ? 1 : TAPS == 3 ? 2 : TAPS == 2 ? (NT == 128 ? 2 : NT == 96 ? 3 : NT == 64 ? 4 : 5)
                                                                  : (NT == 128 ? 4 : NT == 32 ? 7 : 5);
    static constexpr int GA = TAPS == 7 ? 2 : TAPS == 3 ? 3 : TAPS == 2 ? (NT == 128 || NT == 96 ? 3 : NT == 64 ? 4 : 5) : G;
    static constexpr int SEG = TAPS == 7 ? 1 : TAPS == 1 ? 4 : 2;
    static constexpr int BYTES = GA * 3 * (SG_M + (TAPS == 7 ? 56 : TAPS > 1 ? 8 : 0)) * 64 + G * TAPS * 3 * NT * 64;
    static_assert(BYTES + 1024 <= SG_SMEM && GA <= SG_MAX_A && G * TAPS <= SG_MAX_B, "ring");
};

__host__ __device__ inline int sg_hist(int taps, int dil) { return ((taps - 1) * dil + 7) / 8 * 8; }

// Element offset of channel c of row r inside a plane: 64-byte rows, 16-byte chunk index XORed with address bits 7..8.
__host__ __device__ inline long long sg_plane_offset(const SgPlanes& p, int r, int c) {
    return (long long)(c >> 5) * p.group + (long long)r * 32 + ((((c & 31) >> 3) ^ ((r >> 1) & 3)) << 3) + (c & 7);
}

__device__ __forceinline__ void sg_pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void sg_pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// One lane of a converged warp, chosen so that the compiler knows that only one is active: with a comparison of lane numbers it
// wraps every instruction with uniform operands (bulk copies, MMAs, commits) in a loop over the active lanes.
__device__ __forceinline__ bool sg_elect() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}

__device__ __forceinline__ uint32_t sg_smem(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void sg_bar_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sg_smem(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void sg_bar_expect(uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sg_smem(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void sg_bar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sg_smem(bar)) : "memory");
}
__device__ __forceinline__ bool sg_bar_wait(uint64_t* bar, unsigned parity, unsigned limit) {
    const uint32_t a = sg_smem(bar);
    for (unsigned i = 0; i < limit; ++i) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(a), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}
__device__ __forceinline__ void sg_bulk(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(sg_smem(dst)), "l"(src), "r"(bytes), "r"(sg_smem(bar)) : "memory");
}

// Descriptor of a K-major operand tile in 64-byte swizzle (rows 64 bytes apart, 8-row groups 512 bytes apart): the low word holds
// the start address in 16-byte units, the high word is the same for all of them.  The issuing thread adds 32-bit offsets only:
// with 64-bit descriptors and a computed accumulate predicate an MMA cost 65 to 90 cycles to issue, more than it takes to run
// (max(N / 2, 32 + N / 4) cycles for M = 128, K = 16, measured, with no gap between dependent ones).
__device__ __forceinline__ uint32_t sg_desc_lo(uint32_t smem_addr) { return (smem_addr >> 4 & 0x3FFF) | 1u << 16; }
constexpr uint32_t SG_DESC_HI = (512u >> 4) | 1u << 14 | 4u << 29;
// kind::f16: bf16 x bf16 -> fp32, both K-major, M = 128, N = n
__host__ __device__ constexpr uint32_t sg_idesc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(SG_M >> 4) << 24);
}
// One chunk, 32 channels of one tap: ten MMAs.  a, b: low descriptor words of the hi planes; a_plane: distance of the window's
// planes.  The tensor pipe has next to no queue: whatever the issuing thread waits for between two chunks, the pipe waits for too
// (an mbarrier test on a phase long complete: 170 cycles).  So the barriers of the next chunk are tested in front of these MMAs and
// the answers collected behind them, in one asm block; bit 0 of the result: next weights there, with MORE bit 1: next window, bit 2:
// next accumulators free.
template <int NT, bool FIRST, bool MORE>
__device__ __forceinline__ uint32_t sg_chunk(uint32_t d, uint32_t ah, uint32_t bh, uint32_t a_plane, uint32_t bar_b, uint32_t par_b,
                                             uint32_t bar_a, uint32_t par_a, uint32_t bar_t, uint32_t par_t) {
    constexpr uint32_t i1 = sg_idesc(NT), i2 = sg_idesc(2 * NT), bp = NT * 64 >> 4;
    const uint32_t am = ah + a_plane, al = am + a_plane;
    uint32_t ok;
#define SG_TEXT(more_test, more_sel)                                                                                             \
    "{\n\t.reg .pred p, q, r;\n\t.reg .b64 x0, x1, y0, y1, z0, z1, u0, u1, v0, v1, w0, w1;\n\t.reg .b32 t, k;\n\t"                 \
    "mbarrier.test_wait.parity.shared::cta.b64 p, [%11], %12;\n\t" more_test                                                    \
    "mov.b64 x0, {%3, %9};\n\tadd.u32 t, %3, 2;\n\tmov.b64 x1, {t, %9};\n\t"                                                   \
    "mov.b64 y0, {%4, %9};\n\tadd.u32 t, %4, 2;\n\tmov.b64 y1, {t, %9};\n\t"                                                   \
    "mov.b64 z0, {%5, %9};\n\tadd.u32 t, %5, 2;\n\tmov.b64 z1, {t, %9};\n\t"                                                   \
    "mov.b64 u0, {%6, %9};\n\tadd.u32 t, %6, 2;\n\tmov.b64 u1, {t, %9};\n\t"                                                   \
    "mov.b64 v0, {%7, %9};\n\tadd.u32 t, %7, 2;\n\tmov.b64 v1, {t, %9};\n\t"                                                   \
    "mov.b64 w0, {%8, %9};\n\tadd.u32 t, %8, 2;\n\tmov.b64 w1, {t, %9};\n\t"                                                   \
    "tcgen05.mma.cta_group::1.kind::f16 [%1], x0, u0, %10, %17;\n\t"                                                            \
    "tcgen05.mma.cta_group::1.kind::f16 [%2], y0, u0, %18, 1;\n\t"                                                              \
    "tcgen05.mma.cta_group::1.kind::f16 [%2], y0, v0, %18, 1;\n\t"                                                              \
    "tcgen05.mma.cta_group::1.kind::f16 [%2], x0, w0, %18, 1;\n\t"                                                              \
    "tcgen05.mma.cta_group::1.kind::f16 [%2], z0, u0, %18, 1;\n\t"                                                              \
    "tcgen05.mma.cta_group::1.kind::f16 [%1], x1, u1, %10, 1;\n\t"                                                              \
    "tcgen05.mma.cta_group::1.kind::f16 [%2], y1, u1, %18, 1;\n\t"                                                              \
    "tcgen05.mma.cta_group::1.kind::f16 [%2], y1, v1, %18, 1;\n\t"                                                              \
    "tcgen05.mma.cta_group::1.kind::f16 [%2], x1, w1, %18, 1;\n\t"                                                              \
    "tcgen05.mma.cta_group::1.kind::f16 [%2], z1, u1, %18, 1;\n\t"                                                              \
    "selp.u32 %0, 1, 0, p;\n\t" more_sel "}"
#define SG_OPS                                                                                                                   \
    : "=r"(ok)                                                                                                                   \
    : "r"(d), "r"(d + NT), "r"(ah), "r"(am), "r"(al), "r"(bh), "r"(bh + bp), "r"(bh + 2 * bp), "r"(SG_DESC_HI), "r"(i2),          \
      "r"(bar_b), "r"(par_b), "r"(bar_a), "r"(par_a), "r"(bar_t), "r"(par_t), "n"(FIRST ? 0 : 1), "r"(i1)                         \
    : "memory"
    if constexpr (MORE)
        asm volatile(SG_TEXT("mbarrier.test_wait.parity.shared::cta.b64 q, [%13], %14;\n\tmbarrier.test_wait.parity.shared::cta.b64 r, [%15], %16;\n\t",
                             "selp.u32 k, 2, 0, q;\n\tor.b32 %0, %0, k;\n\tselp.u32 k, 4, 0, r;\n\tor.b32 %0, %0, k;\n\t") SG_OPS);
    else
        asm volatile(SG_TEXT("", "") SG_OPS);
#undef SG_TEXT
#undef SG_OPS
    return ok;
}
__device__ __forceinline__ void sg_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(sg_smem(bar)) : "memory");
}
// 16 consecutive columns of this thread's TMEM lane; the caller waits (sg_tmem_wait) before using them
__device__ __forceinline__ void sg_tmem_ld16(uint32_t addr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                   "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(addr));
}
__device__ __forceinline__ void sg_tmem_ld8(uint32_t addr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void sg_tmem_st8(uint32_t addr, const float* v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(addr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
}
__device__ __forceinline__ void sg_tmem_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Eight fp32 values as three 16-byte chunks: v = hi + mid + lo, each rounded to nearest from what is left.
__device__ __forceinline__ void sg_split8(const float (&v)[8], uint4 (&out)[3]) {
    uint32_t w[3][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float a = v[2 * i], b = v[2 * i + 1];
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
            w[p][i] = *reinterpret_cast<const uint32_t*>(&h);
            a -= __low2float(h);
            b -= __high2float(h);
        }
    }
#pragma unroll
    for (int p = 0; p < 3; ++p) out[p] = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
}

__device__ __forceinline__ void sg_split4(const float (&v)[4], uint2 (&out)[3]) {
    const float e[8] = {v[0], v[1], v[2], v[3], 0.f, 0.f, 0.f, 0.f};
    uint4 q[3];
    sg_split8(e, q);
#pragma unroll
    for (int p = 0; p < 3; ++p) out[p] = make_uint2(q[p].x, q[p].y);
}

// Stores eight channels c .. c + 7 (c a multiple of 8) of row r as planes.
__device__ __forceinline__ void sg_store8(const SgPlanes& o, int r, int c, const float (&v)[8]) {
    uint4 q[3];
    sg_split8(v, q);
    bf16* d = o.p + sg_plane_offset(o, r, c);
#pragma unroll
    for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(d + p * o.plane) = q[p];
}

__device__ __forceinline__ float sg_act(float v, int act, float ea, float ib) {
    if (act == SA_SNAKE) { const float s = sinf(v * ea); return v + ib * (s * s); }
    if (act == SA_ELU) {
        // exp(v) - 1 for v <= 0 without a branch: the exponential's own difference below -1/2, its Taylor series above (x^10 / 10! < 3e-10)
        float p = 1.f / 362880.f;
        p = fmaf(p, v, 1.f / 40320.f); p = fmaf(p, v, 1.f / 5040.f); p = fmaf(p, v, 1.f / 720.f); p = fmaf(p, v, 1.f / 120.f);
        p = fmaf(p, v, 1.f / 24.f); p = fmaf(p, v, 1.f / 6.f); p = fmaf(p, v, 0.5f);
        const float near = fmaf(v * v, p, v), far = expf(v) - 1.f;
        return v > 0.f ? v : v > -0.5f ? near : far;
    }
    if (act == SA_GELU) return 0.5f * v * (1.f + erff(v * 0.70710678118654752f));
    return v;
}

// Epilogue of eight consecutive columns n .. n + 7 of row t.  Called in a loop that is not unrolled (the columns come back from
// tensor memory one group at a time): inlined for every column of a thread, the activations make a body that no longer fits the
// instruction caches (an ELU on 128 columns took 172 us for 60 000 rows, 62 us without).  `res_done`: the residual is in v already.
__device__ __forceinline__ void sg_epilogue8(const SgOut& o, float (&v)[8], int n, int t, int M, bool res_done) {
    if (o.gated) {   // four channels; the pairs' other four are the next group's: two 8-byte halves of a chunk
        float u[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) u[j] = (v[2 * j] / (1.f + expf(-v[2 * j]))) * v[2 * j + 1];
        if (t < M) {
            uint2 q[3];
            sg_split4(u, q);
            bf16* d = o.o.p + sg_plane_offset(o.o, o.o.pad + t, n >> 1);
#pragma unroll
            for (int p = 0; p < 3; ++p) *reinterpret_cast<uint2*>(d + p * o.o.plane) = q[p];
        }
        return;
    }
    int c = n, t_out = t, j = 0;
    if (o.up > 1) {           // a column tile lies inside one phase j
        j = n / o.Cout;
        c = n - j * o.Cout;
        t_out = t * o.up + j;
    }
    const int ph = o.p_div > 1 ? t_out % o.p_div : 0, row = o.p_div > 1 ? t_out / o.p_div : t_out;
    SgPlanes op = o.o;
    op.p += (long long)ph * (o.Cout >> 5) * op.group;
    // the rows in front are the next convolution's causal padding: the first rows' threads clear them
    const int zrow = o.up > 1 ? t : row;
    const bool zero = o.o.p && j == 0 && t < SG_PAD && zrow < op.pad;
    if (o.bias) {
        const float4 b0 = __ldg(reinterpret_cast<const float4*>(o.bias + c)), b1 = __ldg(reinterpret_cast<const float4*>(o.bias + c + 4));
        v[0] += b0.x; v[1] += b0.y; v[2] += b0.z; v[3] += b0.w; v[4] += b1.x; v[5] += b1.y; v[6] += b1.z; v[7] += b1.w;
    }
    if (t < M) {
        const long long y0 = ((long long)(c >> 2) * o.y_rows + t_out) * 4, y1 = y0 + 4LL * o.y_rows;
        if (o.res && !res_done) {
            const float4 r0 = __ldcg(reinterpret_cast<const float4*>(o.res + y0)), r1 = __ldcg(reinterpret_cast<const float4*>(o.res + y1));
            float4 s0 = make_float4(1.f, 1.f, 1.f, 1.f), s1 = s0;
            if (o.scale) { s0 = __ldg(reinterpret_cast<const float4*>(o.scale + c)); s1 = __ldg(reinterpret_cast<const float4*>(o.scale + c + 4)); }
            v[0] = r0.x + s0.x * v[0]; v[1] = r0.y + s0.y * v[1]; v[2] = r0.z + s0.z * v[2]; v[3] = r0.w + s0.w * v[3];
            v[4] = r1.x + s1.x * v[4]; v[5] = r1.y + s1.y * v[5]; v[6] = r1.z + s1.z * v[6]; v[7] = r1.w + s1.w * v[7];
        }
        if (o.y && !o.y_act) {
            *reinterpret_cast<float4*>(o.y + y0) = make_float4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<float4*>(o.y + y1) = make_float4(v[4], v[5], v[6], v[7]);
        }
        if (o.act == SA_SNAKE) {
            const float4 e0 = __ldg(reinterpret_cast<const float4*>(o.ea + c)), e1 = __ldg(reinterpret_cast<const float4*>(o.ea + c + 4));
            const float4 i0 = __ldg(reinterpret_cast<const float4*>(o.ib + c)), i1 = __ldg(reinterpret_cast<const float4*>(o.ib + c + 4));
            const float ea[8] = {e0.x, e0.y, e0.z, e0.w, e1.x, e1.y, e1.z, e1.w}, ib[8] = {i0.x, i0.y, i0.z, i0.w, i1.x, i1.y, i1.z, i1.w};
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = sg_act(v[q], SA_SNAKE, ea[q], ib[q]);
        } else if (o.act == SA_ELU) {
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = sg_act(v[q], SA_ELU, 0.f, 0.f);
        } else if (o.act == SA_GELU) {
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = sg_act(v[q], SA_GELU, 0.f, 0.f);
        }
        if (o.y && o.y_act) {
            *reinterpret_cast<float4*>(o.y + y0) = make_float4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<float4*>(o.y + y1) = make_float4(v[4], v[5], v[6], v[7]);
        }
        if (o.o.p) sg_store8(op, op.pad + row, c, v);
    }
    if (zero) {
        bf16* d = op.p + sg_plane_offset(op, zrow, c);
#pragma unroll
        for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(d + p * op.plane) = make_uint4(0, 0, 0, 0);
    }
}

template <int NT, int TAPS>
__global__ void __launch_bounds__(SG_THREADS, 1) k_sg(const __grid_constant__ SgArgs a) {
    extern __shared__ unsigned char sg_dyn[];
    __shared__ uint64_t a_full[SG_MAX_A], a_empty[SG_MAX_A], b_full[SG_MAX_B], b_empty[SG_MAX_B], t_full[2], t_empty[2];
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_bad;
    constexpr int NC = NT / 2;                                            // columns of an epilogue thread
    // two pairs of accumulators and, where there is room, NT columns in which a finished tile waits for its epilogue
    constexpr bool STASH = NT < 128;
    constexpr uint32_t TMEM_COLS = NT == 32 ? 256 : 512;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    using R = SgRing<NT, TAPS>;
    const int hist = sg_hist(TAPS, a.dil), W = SG_M + hist, shift0 = hist - (TAPS - 1) * a.dil;
    const uint32_t a_bytes = 3u * W * 64u, b_bytes = 3u * NT * 64u;
    unsigned char* sA = sg_dyn + ((1024u - (sg_smem(sg_dyn) & 1023u)) & 1023u);
    unsigned char* sB = sA + (size_t)R::GA * a_bytes;
    if (tid == 0) {
        for (int i = 0; i < SG_MAX_A; ++i) { sg_bar_init(&a_full[i], 1); sg_bar_init(&a_empty[i], 1); }
        for (int i = 0; i < SG_MAX_B; ++i) { sg_bar_init(&b_full[i], 1); sg_bar_init(&b_empty[i], 1); }
        for (int i = 0; i < 2; ++i) { sg_bar_init(&t_full[i], 1); sg_bar_init(&t_empty[i], SG_EPI_WARPS); }
        s_bad = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 3) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sg_smem(&s_tmem)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    sg_pdl_launch();   // every CTA of this grid owns its tensor memory by now
    const int tiles = a.m_tiles * a.n_tiles, S = a.splits;
    const int rank = S > 1 ? blockIdx.x % S : 0;                       // a cluster's CTAs share a tile, each a range of channels
    const int kc0 = rank * a.kchunks / S, kchunks = (rank + 1) * a.kchunks / S - kc0, chunks = kchunks * TAPS;
    const int tile0 = blockIdx.x / S, tile_step = S > 1 ? tiles : gridDim.x;
    unsigned limit = a.spin_limit;
    auto wait = [&](uint64_t* bar, unsigned parity) {
        if (sg_bar_wait(bar, parity, limit)) return;
        limit = 16;   // after its first expired wait a thread walks the rest of its sequence without waiting
        s_bad = 1;
    };

    if (warp == 0) {
        if (sg_elect()) {
            sg_pdl_wait();
            int st = 0;
            unsigned ph = 1;
            bool filled = false;
            for (int tile = tile0; tile < tiles; tile += tile_step) {
                const int m = tile / a.n_tiles;
                const bf16* src = a.x.p + (long long)(a.x.pad - hist + m * SG_M) * 32;
                for (int kc = 0; kc < kchunks; ++kc) {
                    if (filled) wait(&a_empty[st], ph);
                    sg_bar_expect(&a_full[st], a_bytes);
                    const bf16* g = src + (kc0 + kc) * a.x.group;
                    unsigned char* d = sA + (size_t)st * a_bytes;
                    sg_bulk(d, g, a_bytes / 3, &a_full[st]);
                    sg_bulk(d + a_bytes / 3, g + a.x.plane, a_bytes / 3, &a_full[st]);
                    sg_bulk(d + a_bytes / 3 * 2, g + 2 * a.x.plane, a_bytes / 3, &a_full[st]);
                    if (++st == R::GA) { st = 0; ph ^= 1; filled = true; }
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (sg_elect()) {
            int st = 0;
            unsigned ph = 1;
            bool filled = false;
            for (int tile = tile0; tile < tiles; tile += tile_step) {
                const unsigned char* src = reinterpret_cast<const unsigned char*>(a.w) +
                                           ((size_t)(tile % a.n_tiles) * a.kchunks + kc0) * TAPS * b_bytes;
                for (int c = 0; c < chunks; ++c) {
                    if (filled) wait(&b_empty[st], ph);
                    sg_bar_expect(&b_full[st], b_bytes);
                    sg_bulk(sB + (size_t)st * b_bytes, src + (size_t)c * b_bytes, b_bytes, &b_full[st]);
                    if (++st == R::G * TAPS) { st = 0; ph ^= 1; filled = true; }
                }
                if (a.b_keep) break;
            }
        }
        __syncwarp();
    } else if (warp == 2) {
        if (sg_elect()) {
            sg_pdl_wait();   // the windows come behind the dependency: its wait is not this thread's barriers' to count
            const uint32_t a_plane = a_bytes / 3 >> 4, a0 = sg_desc_lo(sg_smem(sA)) + shift0 * 4, b0 = sg_desc_lo(sg_smem(sB));
            int sa = 0, sb = 0, seg = 0, left = 0;      // slots, segments so far, channel groups left in this one
            uint32_t pa = 0, pb = 0, ok = 0, d = 0, fb = 0;   // parities, what is known to be complete, accumulators, first weight stage
            for (int tile = tile0; tile < tiles; tile += tile_step) {
                if (a.b_keep) sb = 0;                   // the kept stages' phase 0 stays complete
                for (int kc = 0; kc < kchunks; ++kc) {
                    const bool first = left == 0;
                    if (first) {
                        if (!(ok & 4) && seg >= 2) wait(&t_empty[seg & 1], ((seg >> 1) & 1) ^ 1);
                        d = tmem + (seg & 1) * 2 * NT;
                        left = min(R::SEG, kchunks - kc);
                    }
                    --left;
                    if (!(ok & 2)) wait(&a_full[sa], pa);
                    const uint32_t da = a0 + sa * (a_bytes >> 4);
                    uint64_t* const a_done = &a_empty[sa];
                    fb = sb * TAPS;
                    const uint32_t db = b0 + fb * (b_bytes >> 4), bars = sg_smem(&b_full[fb]), p0 = pb;
                    if (++sa == R::GA) { sa = 0; pa ^= 1; }
                    if (++sb == R::G && !a.b_keep) { sb = 0; pb ^= 1; }
                    const uint32_t next_b = sg_smem(&b_full[sb * TAPS < R::G * TAPS ? sb * TAPS : 0]), next_a = sg_smem(&a_full[sa]), next_t = sg_smem(&t_empty[(seg & 1) ^ 1]);
                    const uint32_t par_t = (((seg + 1) >> 1) & 1) ^ 1;
#pragma unroll
                    for (int tap = 0; tap < TAPS; ++tap) {
                        if (!(ok & 1)) wait(&b_full[fb + tap], p0);
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const uint32_t x = da + tap * a.dil * 4, y = db + tap * (b_bytes >> 4), nb = tap == TAPS - 1 ? next_b : bars + 8 * (tap + 1), np = tap == TAPS - 1 ? pb : p0;
                        if (tap == 0 && first) ok = sg_chunk<NT, true, TAPS == 1>(d, x, y, a_plane, nb, np, next_a, pa, next_t, par_t);
                        else if (tap == TAPS - 1) ok = sg_chunk<NT, false, true>(d, x, y, a_plane, nb, np, next_a, pa, next_t, par_t);
                        else ok = sg_chunk<NT, false, false>(d, x, y, a_plane, nb, np, next_a, pa, next_t, par_t);
                        sg_commit(&b_empty[fb + tap]);
                    }
                    sg_commit(a_done);
                    if (left == 0) sg_commit(&t_full[seg++ & 1]);
                }
            }
        }
        __syncwarp();
    } else if (warp >= 4) {
        const int quarter = warp & 3, half = (warp - 4) >> 2;
        const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16) + half * NC;
        const int n_seg = (kchunks + R::SEG - 1) / R::SEG;
        const int part = half * 4 + quarter, per = SG_EPI_WARPS / S, owner = part / per;   // CTA r of a split tile finishes parts [r per, (r + 1) per)
        int seg = 0;
        sg_pdl_wait();   // the residual is read, and the outputs' buffers may still be read by earlier launches
        for (int tile = tile0; tile < tiles; tile += tile_step) {
            const int m = tile / a.n_tiles, n0 = (tile - m * a.n_tiles) * NT + half * NC, t = m * SG_M + quarter * 32 + lane;
            float acc[NC];
            // a residual without a scale is where the sum starts: all its loads are in flight while the MMAs run
            const bool res_first = a.out.res && !a.out.scale && a.out.up == 1 && owner == rank;
            if (res_first && t < a.M) {
#pragma unroll
                for (int i = 0; i < NC; i += 4) {
                    const float4 r = __ldcg(reinterpret_cast<const float4*>(a.out.res + ((long long)((n0 + i) >> 2) * a.out.y_rows + t) * 4));
                    acc[i] = r.x; acc[i + 1] = r.y; acc[i + 2] = r.z; acc[i + 3] = r.w;
                }
            } else {
#pragma unroll
                for (int i = 0; i < NC; ++i) acc[i] = 0.f;
            }
            for (int s = 0; s < n_seg; ++s, ++seg) {
                const int buf = seg & 1;
                wait(&t_full[buf], (seg >> 1) & 1);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                __syncwarp();
                const uint32_t d = lane_base + buf * 2 * NT;
#pragma unroll
                for (int i = 0; i < NC; i += 16) {
                    uint32_t hi[16], lo[16];
                    sg_tmem_ld16(d + i, hi);
                    sg_tmem_ld16(d + NT + i, lo);
                    sg_tmem_wait();
#pragma unroll
                    for (int q = 0; q < 16; ++q) acc[i + q] += __uint_as_float(hi[q]) + __uint_as_float(lo[q]);
                }
                if (STASH || s + 1 < n_seg) {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) sg_bar_arrive(&t_empty[buf]);
                }
            }
            if (S > 1) {
                // partial sums to the CTA that finishes this part, then added there in rank order.  They land in its ring: behind the
                // first barrier every CTA's MMAs, and with them all use of the rings, are over.
                asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
                __syncwarp();
                float* const mail = reinterpret_cast<float*>(sA) + ((part % per) * (NC / 4) * 32 + lane) * 4;
                const int slot_stride = per * NC * 32;
                if (owner != rank) {
                    const uint32_t dst = sg_smem(mail + (rank < owner ? rank : rank - 1) * slot_stride);
#pragma unroll
                    for (int i = 0; i < NC; i += 4)
                        asm volatile("{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %0, %1;\n\tst.shared::cluster.v4.f32 [r], {%2, %3, %4, %5};\n\t}"
                                     ::"r"(dst + i * 128), "r"(owner), "f"(acc[i]), "f"(acc[i + 1]), "f"(acc[i + 2]), "f"(acc[i + 3]) : "memory");
                }
                asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
                __syncwarp();
                if (owner != rank) break;
                for (int slot = 0; slot < S - 1; ++slot) {
#pragma unroll
                    for (int i = 0; i < NC; i += 4) {
                        const float4 p = *reinterpret_cast<const float4*>(mail + slot * slot_stride + i * 32);
                        acc[i] += p.x; acc[i + 1] += p.y; acc[i + 2] += p.z; acc[i + 3] += p.w;
                    }
                }
            }
            // the sums go back to tensor memory, so that the loop below can fetch them by address
            const uint32_t d = lane_base + (STASH ? 4 * NT : ((seg - 1) & 1) * 2 * NT);
#pragma unroll
            for (int i = 0; i < NC; i += 8) sg_tmem_st8(d + i, acc + i);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
#pragma unroll 1
            for (int i = 0; i < NC; i += 8) {
                float v[8];
                sg_tmem_ld8(d + i, v);
                sg_epilogue8(a.out, v, n0 + i, t, a.M, res_first);
            }
            if (!STASH) {
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) sg_bar_arrive(&t_empty[(seg - 1) & 1]);
            }
        }
    }
    if (S > 1 && warp < 4)
        asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;\n\tbarrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (s_bad && tid == 0) {   // gave up somewhere: what may still be on its way to this CTA's shared memory lands before it retires
        atomicOr(a.flag, SG_FLAG_WAIT);
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    }
    if (warp == 3) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
}

// ---------------------------------------------------------------- weights
// Where element (column n, tap, input channel c) of a packed matrix comes from.
enum {
    SW_ROWS = 0,     // w[n][c][taps]: a matrix, or a convolution of stride 1 in torch's layout
    SW_STRIDED,      // w[n][c'][2 s], s = q0, C = q1: tap = k / s, c = (k % s) * C + c'
    SW_TR_ROWS,      // transposed, w[(co, k)][c], k < 2 s, s = q0, Cout = q1: column (j, co), tap 0 (row t - 1) k = j + s, tap 1 k = j
    SW_TR_TILES,     // the same, rows in tiles of 96: w[row / 96][c][row % 96]
    SW_TILES,        // w[n / 96][c][taps][n % 96]
    SW_PAIR,         // gated pair: columns 2 i from w, 2 i + 1 from w2, rows of C
    SW_CAT           // w[n][C / 2] | w2[n][C / 2] side by side
};

struct SgPack {
    const float* w;
    const float* w2;
    bf16* out;
    int mode, q0, q1;
    int N, C, taps, NT;
};

__device__ __forceinline__ float sg_weight(const SgPack& a, int n, int tap, int c) {
    switch (a.mode) {
        case SW_STRIDED: return a.w[((long long)n * a.q1 + c % a.q1) * (2 * a.q0) + tap * a.q0 + c / a.q1];
        case SW_TR_ROWS:
        case SW_TR_TILES: {
            // (kernel = stride: one tap, k = j)
            const int j = n / a.q1, co = n - j * a.q1, row = a.taps == 1 ? co * a.q0 + j : co * 2 * a.q0 + (tap == 0 ? j + a.q0 : j);
            return a.mode == SW_TR_ROWS ? a.w[(long long)row * a.C + c] : a.w[((long long)(row / 96) * a.C + c) * 96 + row % 96];
        }
        case SW_TILES: return a.w[(((long long)(n / 96) * a.C + c) * a.taps + tap) * 96 + n % 96];
        case SW_PAIR: return (n & 1 ? a.w2 : a.w)[(long long)(n >> 1) * a.C + c];
        case SW_CAT: return c < a.C / 2 ? a.w[(long long)n * (a.C / 2) + c] : a.w2[(long long)n * (a.C / 2) + c - a.C / 2];
        default: return a.w[((long long)n * a.C + c) * a.taps + tap];
    }
}

// One thread per eight channels of a (column, tap): three 16-byte chunks of the stage image.
static __global__ void __launch_bounds__(256) k_sg_pack(SgPack a) {
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    const int groups = a.C / 8;
    if (i >= (long long)a.N * a.taps * groups) return;
    const int g = (int)(i % groups), tap = (int)(i / groups % a.taps), n = (int)(i / groups / a.taps);
    float v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = sg_weight(a, n, tap, g * 8 + q);
    uint4 out[3];
    sg_split8(v, out);
    const int r = n % a.NT, kc = g >> 2, chunk = g & 3;
    bf16* d = a.out + (((long long)(n / a.NT) * (a.C / 32) + kc) * a.taps + tap) * 3 * a.NT * 32;
#pragma unroll
    for (int p = 0; p < 3; ++p)
        *reinterpret_cast<uint4*>(d + ((long long)p * a.NT + r) * 32 + ((chunk ^ ((r >> 1) & 3)) << 3)) = out[p];
}

// A packed matrix and the shape its launches need.
struct SgWeight {
    const bf16* p;
    int N, C, taps, NT;
};

inline size_t sg_weight_bytes(int N, int C, int taps) { return (size_t)N * C * taps * 6; }

inline cudaError_t sg_pack(const SgPack& a, cudaStream_t s) {
    const long long n = (long long)a.N * a.taps * (a.C / 8);
    k_sg_pack<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a);
    return cudaGetLastError();
}

// What the launches of a sequence share.
struct SgCtx {
    int* flag;
    int num_sms;
    bool pdl;
    cudaStream_t s;
    int64_t* launches;
};

template <class... KArgs, class... Args>
cudaError_t sg_run(const SgCtx& x, void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, const Args&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = x.s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = x.pdl ? 1 : 0;
    ++*x.launches;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

template <class... KArgs, class... Args>
cudaError_t sg_run_cluster(const SgCtx& x, void (*kern)(KArgs...), int cluster, dim3 grid, dim3 block, size_t smem, const Args&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = x.s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = x.pdl ? 2 : 1;
    ++*x.launches;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

template <int NT, int TAPS>
cudaError_t sg_launch_nt(const SgCtx& x, SgArgs a) {
    const int tiles = a.m_tiles * a.n_tiles;
    int grid = tiles < x.num_sms ? tiles : x.num_sms;
    a.splits = 1;
    // Few tiles (125 rows of 512 columns are 16): a cluster of CTAs shares the channels of each, as long as every one has at least
    // eight chunks (about 4 us of weights to fetch; the exchange costs 2) and all are resident at once (15 clusters of eight).
    for (int s = 2; s <= 8; s *= 2)
        if (tiles * s <= (s == 8 ? 120 : x.num_sms) && a.kchunks >= 2 * s && a.kchunks * TAPS >= 8 * s) a.splits = s;
    if (a.splits > 1) grid = tiles * a.splits;
    else if (tiles > grid && a.kchunks <= SgRing<NT, TAPS>::G && a.n_tiles <= grid) {
        a.b_keep = 1;
        grid -= grid % a.n_tiles;   // a CTA's tiles then have the same column tile
    }
    static thread_local int ready = -1;   // device whose copy of the kernel this thread has opted into its shared memory
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess && ready != dev) {
        e = cudaFuncSetAttribute(k_sg<NT, TAPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, SG_SMEM);
        ready = dev;
    }
    if (e != cudaSuccess) return e;
    if (a.splits == 1) return sg_run(x, k_sg<NT, TAPS>, dim3(grid), dim3(SG_THREADS), SG_SMEM, a);
    return sg_run_cluster(x, k_sg<NT, TAPS>, a.splits, dim3(grid), dim3(SG_THREADS), SG_SMEM, a);
}

// D = X (*) W over M rows.  out.up / out.Cout describe the columns; N = W.N must be a multiple of W.NT.
inline cudaError_t sg_launch(const SgCtx& ctx, const SgWeight& w, const SgPlanes& x, int M, int dil, const SgOut& out) {
    SgArgs a = {};
    a.x = x; a.w = w.p; a.kchunks = w.C / 32; a.dil = dil; a.M = M;
    a.n_tiles = w.N / w.NT; a.m_tiles = (M + SG_M - 1) / SG_M;
    a.out = out; a.flag = ctx.flag; a.spin_limit = SG_SPIN_LIMIT;
    const int hist = sg_hist(w.taps, dil);
    if (w.N % w.NT || w.C % 32 || M < 1 || x.pad % 8 || x.pad < hist || hist > (w.taps == 7 ? 56 : 8) || (out.up > 1 && out.Cout % w.NT)) return cudaErrorInvalidValue;
    switch (w.taps * 1000 + w.NT) {
        case 1032: return sg_launch_nt<32, 1>(ctx, a);
        case 1064: return sg_launch_nt<64, 1>(ctx, a);
        case 1096: return sg_launch_nt<96, 1>(ctx, a);
        case 1128: return sg_launch_nt<128, 1>(ctx, a);
        case 2032: return sg_launch_nt<32, 2>(ctx, a);
        case 2064: return sg_launch_nt<64, 2>(ctx, a);
        case 2096: return sg_launch_nt<96, 2>(ctx, a);
        case 2128: return sg_launch_nt<128, 2>(ctx, a);
        case 3032: return sg_launch_nt<32, 3>(ctx, a);
        case 3064: return sg_launch_nt<64, 3>(ctx, a);
        case 7064: return sg_launch_nt<64, 7>(ctx, a);
        case 7096: return sg_launch_nt<96, 7>(ctx, a);
        default: return cudaErrorInvalidValue;
    }
}

// Rows a plane buffer for T rows of time needs: the padding in front and whole tiles behind.
inline int sg_rows(int T, int pad) { return pad + (T + SG_M - 1) / SG_M * SG_M; }

inline size_t sg_plane_bytes(int C, int T, int pad) { return (size_t)3 * C * sg_rows(T, pad) * 2; }

inline SgPlanes sg_planes(void* p, int C, int T, int pad) {
    SgPlanes o;
    o.p = static_cast<bf16*>(p);
    o.pad = pad;
    o.group = (long long)sg_rows(T, pad) * 32;
    o.plane = o.group * (C / 32);
    return o;
}

}  // namespace vuis
