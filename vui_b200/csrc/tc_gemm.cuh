// GEMM for several streams and for prefill rows on the 5th-generation tensor cores:
//   D[n][m] = sum_k W[n][k] * X[m][k]      (W: weights (N, K) bf16; X: activations (M, K) bf16)
// "swap-AB": a tile of 128 weight rows is the MMA's M side, MT = 16 .. 128 activation rows its N side, so one tcgen05.mma covers
// every stream of the tile and each weight byte is read once per row block.
//
//  * operands reach shared memory through TMA (cp.async.bulk.tensor.2d, 128-byte swizzle, K-major), one elected thread issues
//    tcgen05.mma (kind::f16, bf16 x bf16 -> fp32; max(MT / 2, 32 + MT / 4) cycles per 16 of K), the accumulator tile lives in tensor
//    memory and is read back with tcgen05.ld; an mbarrier ring decouples the two;
//  * few tiles leave most SMs idle, so the CTAs of a cluster (2 or 4) share a tile's K.  Each sends its partial rows to the CTA
//    that finishes them (st.async into the owner's shared memory, counted on its mbarrier: one hop), which adds them in a
//    fixed order and runs the epilogue functor (RoPE + KV append, residual add, SwiGLU, logits).  Through global memory and a
//    counter the exchange took 5 us of a GEMM's 9;
//  * launched with programmatic dependent launch: the weight tiles of the first stages are requested before the kernel waits for
//    its predecessor, the activations after.
// Every wait is bounded and records FLAG_TC_TIMEOUT instead of hanging.  No TMA load here uses cluster multicast.
#pragma once
#include <cuda.h>

#include "decode_kernels.cuh"

namespace vuib {

constexpr int TC_THREADS = 256;
constexpr int TC_TILE_N = 128;      // weight rows per CTA
constexpr int TC_BOX_N = 64;        // rows of a TMA box of weights (PAIRED: 16, w1 and w3 in turn)
constexpr int TC_KCHUNK = 64;       // bf16 per row per stage = 128 bytes = one swizzle span
constexpr int TC_MAX_STAGES = 12;     // ring depth is set per launch from the shared memory left
constexpr int TC_MAX_M = 128;            // most activation rows of a tile
constexpr int TC_EPI_BYTES_PER_M = 256, TC_EPI_HEAD = TC_MAX_M * 8;  // epilogue staging: 128 bf16 per activation row behind a number each
constexpr int FLAG_TC_TIMEOUT = 16;
constexpr unsigned TC_SPIN_LIMIT = 1u << 22;  // default bound of every wait below, in polls (TcArgs::spin_limit)

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

// Bounded wait on a phase parity; returns false after `limit` probes.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity, unsigned limit) {
    const uint32_t a = smem_u32(bar);
    for (unsigned spins = 0; spins < limit; ++spins) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(a), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_u32(smem_dst)), "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

// One lane of a converged warp, chosen so that the compiler knows that only one is active: with a comparison of lane numbers it
// wraps every instruction with uniform operands (TMA copies, MMAs, commits) in a loop over the active lanes.
__device__ __forceinline__ bool tc_elect() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}

// Descriptor of a K-major, 128-byte-swizzled operand tile (rows 128 bytes apart, 8-row groups 1024): the low word holds the start
// address in 16-byte units, the high word is the same for all.  The issuing thread adds 32-bit offsets only: the tensor pipe has
// next to no queue, so that what it spends on 64-bit descriptors and predicates the pipe waits for too.
__device__ __forceinline__ uint32_t tc_desc(const void* smem) { return (smem_u32(smem) >> 4 & 0x3FFF) | 1u << 16; }
constexpr uint32_t TC_DESC_HI = (1024u >> 4) | 1u << 14 | 2u << 29;
// kind::f16 instruction descriptor: bf16 A and B, fp32 accumulate, both K-major, M = 128, N = n.
__host__ __device__ constexpr uint32_t tc_idesc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | (8u << 24);
}

// 64 of K for one tile: four MMAs.  With TEST the barrier of the next stage is tested in front of them and the answer collected
// behind (a test's 170 cycles would otherwise be the tensor pipe's too).
template <bool FIRST, bool TEST>
__device__ __forceinline__ uint32_t tc_mma4(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t bar, uint32_t parity) {
    uint32_t ok = 0;
#define TC_BODY(pre, post)                                                                                                        \
    "{\n\t.reg .pred p;\n\t.reg .b64 x, y;\n\t.reg .b32 t, u;\n\t" pre                                                              \
    "mov.b64 x, {%2, %4};\n\tmov.b64 y, {%3, %4};\n\ttcgen05.mma.cta_group::1.kind::f16 [%1], x, y, %5, %8;\n\t"                     \
    "add.u32 t, %2, 2;\n\tadd.u32 u, %3, 2;\n\tmov.b64 x, {t, %4};\n\tmov.b64 y, {u, %4};\n\ttcgen05.mma.cta_group::1.kind::f16 [%1], x, y, %5, 1;\n\t" \
    "add.u32 t, %2, 4;\n\tadd.u32 u, %3, 4;\n\tmov.b64 x, {t, %4};\n\tmov.b64 y, {u, %4};\n\ttcgen05.mma.cta_group::1.kind::f16 [%1], x, y, %5, 1;\n\t" \
    "add.u32 t, %2, 6;\n\tadd.u32 u, %3, 6;\n\tmov.b64 x, {t, %4};\n\tmov.b64 y, {u, %4};\n\ttcgen05.mma.cta_group::1.kind::f16 [%1], x, y, %5, 1;\n\t" \
    post "}"
#define TC_OPS : "=r"(ok) : "r"(d), "r"(a), "r"(b), "r"(TC_DESC_HI), "r"(idesc), "r"(bar), "r"(parity), "n"(FIRST ? 0 : 1) : "memory"
    if constexpr (TEST)
        asm volatile(TC_BODY("mbarrier.test_wait.parity.shared::cta.b64 p, [%6], %7;\n\t", "selp.u32 %0, 1, 0, p;\n\t") TC_OPS);
    else
        asm volatile(TC_BODY("", "mov.u32 %0, 0;\n\t") TC_OPS);
#undef TC_BODY
#undef TC_OPS
    return ok;
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                   "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// 32 consecutive accumulator columns of this thread's TMEM lane in one instruction.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// x / (1 + exp(-x)) as (x or x exp(x)) / (1 + exp(-|x|)): the divisor lies in [1, 2], so that CUDA's branch-free __fdividef is within
// its two ulp for every x.
__device__ __forceinline__ float silu(float x) {
    const float e = expf(-fabsf(x));
    return __fdividef(x < 0.f ? x * e : x, 1.0f + e);
}

// ---------------------------------------------------------------------------
// Epilogue functors.  A thread owns weight row n (0..127 of the tile) and is handed
// 8 consecutive activation rows m0..m0+7 at a time (the whole CTA calls together).
// ---------------------------------------------------------------------------
struct TcEpiQkv {      // RoPE on q,k + K/V append (EpiQkv of the GEMV path)
    bf16* q_out; int q_cols, kv_cols;
    bf16* k_cache; bf16* v_cache;
    const int32_t* row_slot; const int32_t* row_pos; int max_seq;
    const bf16* rope;
    int rows_per_b, pos_base;
    int m_off;  // row index of m = 0 in the depth-transformer addressing
    static constexpr bool PAIRED = false;
    static constexpr bool STAGED = true;
    // While the MMAs run: the cache row of every activation row, and the RoPE rows [cos,sin] x 64 of its position -> es[m][128].  (With
    // slot and position read in apply() a round trip to the L2 stood in front of every eight rows' stores.)
    __device__ __forceinline__ void stage(unsigned char* es, int tile, int M, int tid) const {
        if (tid < M) {
            const int slot = row_slot ? __ldcg(row_slot + tid) : (tid + m_off) / rows_per_b;
            const int pos = row_slot ? __ldcg(row_pos + tid) : pos_base + (tid + m_off) % rows_per_b;
            reinterpret_cast<long long*>(es)[tid] = (long long)slot * max_seq + pos;
        }
        if (!rope) return;
        uint4* dst = reinterpret_cast<uint4*>(es + TC_EPI_HEAD);
#pragma unroll 4
        for (int i = tid; i < M * 16; i += TC_THREADS) {
            const int m = i >> 4, c = i & 15;
            const int pos = row_slot ? __ldcg(row_pos + m) : pos_base + (m + m_off) % rows_per_b;
            dst[i] = __ldg(reinterpret_cast<const uint4*>(rope + (size_t)pos * HD * 2) + c);
        }
    }
    __host__ __device__ TcEpiQkv shifted(int m) const {
        TcEpiQkv o = *this;
        o.q_out += (size_t)m * q_cols;
        if (row_slot) { o.row_slot += m; o.row_pos += m; }
        o.m_off += m;
        return o;
    }
    __device__ __forceinline__ void apply(int n, int m0, int M, const float (&v)[8], float*,
                                          const unsigned char* es) const {
        const bool odd = n & 1;
        const bool do_rope = rope && n < q_cols + kv_cols;
        const bool to_cache = n >= q_cols;
        const long long* cache_row = reinterpret_cast<const long long*>(es);
        const __nv_bfloat162* rs = reinterpret_cast<const __nv_bfloat162*>(es + TC_EPI_HEAD);
        bf16* const out = !to_cache ? q_out + n : n < q_cols + kv_cols ? k_cache + (n - q_cols) : v_cache + (n - q_cols - kv_cols);
        float t[8], other[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) t[j] = rbf(v[j]);
#pragma unroll
        for (int j = 0; j < 8; ++j) other[j] = __shfl_xor_sync(0xffffffffu, t[j], 1);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int m = m0 + j, mm = min(m, M - 1);
            if (do_rope) {
                const __nv_bfloat162 f = rs[mm * 64 + (n & (HD - 1))];
                const float c = __low2float(f), sn = odd ? __high2float(f) : -__high2float(f);
                t[j] = rbf(rbf(t[j] * c) + rbf(other[j] * sn));
            }
            const size_t at = to_cache ? (size_t)cache_row[mm] * kv_cols : (size_t)m * q_cols;
            if (m < M) out[at] = f2bf(t[j]);
        }
    }
};

struct TcEpiResidual {  // x += bf16(acc)
    bf16* x; int N; bf16* tap;
    static constexpr bool PAIRED = false;
    static constexpr bool STAGED = true;
    // While the MMAs run: this tile's slice of the residual stream, x[m][tile*128 .. +128) -> es[m][128].
    __device__ __forceinline__ void stage(unsigned char* es, int tile, int M, int tid) const {
        uint4* dst = reinterpret_cast<uint4*>(es);
#pragma unroll 4
        for (int i = tid; i < M * 16; i += TC_THREADS) {
            const int m = i >> 4, c = i & 15;
            dst[i] = __ldcg(reinterpret_cast<const uint4*>(x + (size_t)m * N + tile * TC_TILE_N) + c);
        }
    }
    __host__ __device__ TcEpiResidual shifted(int m) const {
        TcEpiResidual o = *this;
        o.x += (size_t)m * N;
        if (tap) o.tap += (size_t)m * N;
        return o;
    }
    __device__ __forceinline__ void apply(int n, int m0, int M, const float (&v)[8], float*,
                                          const unsigned char* es) const {
        const bf16* xs = reinterpret_cast<const bf16*>(es);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int m = m0 + j;
            if (m >= M) continue;
            const size_t idx = (size_t)m * N + n;
            const bf16 o = f2bf(bf2f(xs[m * TC_TILE_N + (n & (TC_TILE_N - 1))]) + rbf(v[j]));
            x[idx] = o;
            if (tap) tap[idx] = o;
        }
    }
};

struct TcEpiSwiGLU {    // of every 32 tile rows, 16 are w1 rows and 16 the same hidden units' w3 rows
    bf16* act; int F;
    static constexpr bool PAIRED = true;
    static constexpr bool STAGED = false;
    __host__ __device__ TcEpiSwiGLU shifted(int m) const {
        TcEpiSwiGLU o = *this;
        o.act += (size_t)m * F;
        return o;
    }
    // a1 = the unit's w1 sums, a3 = its w3 sums, for activation rows m0 .. m0 + 3
    __device__ __forceinline__ void apply_pair(int unit, int m0, int M, const float (&a1)[4], const float (&a3)[4]) const {
        bf16 o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) o[j] = f2bf(rbf(silu(rbf(a1[j]))) * rbf(a3[j]));
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (m0 + j < M) act[(size_t)(m0 + j) * F + unit] = o[j];
    }
};

struct TcEpiLogits {    // plain bf16 rows (+ optional second copy with its own stride)
    bf16* out; int N; bf16* tap; int tap_stride;
    static constexpr bool PAIRED = false;
    static constexpr bool STAGED = false;
    __host__ __device__ TcEpiLogits shifted(int m) const {
        TcEpiLogits o = *this;
        o.out += (size_t)m * N;
        if (tap) o.tap += (size_t)m * tap_stride;
        return o;
    }
    __device__ __forceinline__ void apply(int n, int m0, int M, const float (&v)[8], float*,
                                          const unsigned char*) const {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int m = m0 + j;
            if (m >= M) continue;
            const bf16 o = f2bf(v[j]);
            out[(size_t)m * N + n] = o;
            if (tap) tap[(size_t)m * tap_stride + n] = o;
        }
    }
};

struct TcEpiProjPos {   // depth position 0: bf16(acc) + pos_emb[0], written to row m*row_mul
    const bf16* pos_emb; bf16* out; int rd, row_mul;
    static constexpr bool PAIRED = false;
    static constexpr bool STAGED = false;
    __host__ __device__ TcEpiProjPos shifted(int m) const {
        TcEpiProjPos o = *this;
        o.out += (size_t)m * row_mul * rd;
        return o;
    }
    __device__ __forceinline__ void apply(int n, int m0, int M, const float (&v)[8], float*,
                                          const unsigned char*) const {
        const float pe = bf2f(pos_emb[n]);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int m = m0 + j;
            if (m >= M) continue;
            out[(size_t)m * row_mul * rd + n] = f2bf(rbf(v[j]) + pe);
        }
    }
};

struct TcArgs {
    int row_off;      // first weight row of tile 0 inside the mapped matrix (stacked depth heads)
    int M, MT;        // activation rows in all; rows of a tile, 16 to 128: the grid's z dimension walks blocks of MT rows
    int chunks;       // K chunks of 64 in all; CTA s of a cluster handles chunks [s*chunks/splits, (s+1)*chunks/splits)
    int stages;       // TMA ring depth (<= TC_MAX_STAGES, <= the shortest split)
    int splits;       // gridDim.x = CTAs of a cluster: 1, 2 or 4
    int segs;         // accumulators per CTA: 1, 2 or 4 equal parts of its chunks, added pairwise (see tc_gemm in vuib200.cu)
    int withhold;     // test hook: the first CTA expects one value more than is sent to it
    int32_t* flag;
    unsigned long long* dbg;  // optional: device-clock stamps of CTA (0,0) (profiling aid)
    unsigned spin_limit;      // polls after which a wait gives up and records FLAG_TC_TIMEOUT
};

__device__ __forceinline__ void tc_stamp(const TcArgs& a, int i) {
    if (a.dbg && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && threadIdx.x == 64) {
        unsigned long long t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        a.dbg[i] = t;
    }
}

// Eight sums of tile row `row` (n = tile * 128 + row) for activation rows m0 .. m0 + 7.  PAIRED: lanes l and l + 16 hold one unit's w1
// and w3 sums; the lower one takes the first four activation rows, the upper one the others.
template <class Epi>
__device__ __forceinline__ void tc_apply(const Epi& ep, int tile, int row, int m0, int M, const float (&v)[8], const unsigned char* es) {
    if constexpr (Epi::PAIRED) {
        const bool low = (row & 16) == 0;
        float a1[4], a3[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float got = __shfl_xor_sync(0xffffffffu, low ? v[j + 4] : v[j], 16);
            a1[j] = low ? v[j] : got;
            a3[j] = low ? got : v[j + 4];
        }
        ep.apply_pair(tile * 64 + (row >> 5) * 16 + (row & 15), low ? m0 : m0 + 4, M, a1, a3);
    } else {
        ep.apply(tile * TC_TILE_N + row, m0, M, v, nullptr, es);
    }
}

// N columns of this thread's row, the sum of Q accumulators MT columns apart, added as a balanced tree.
template <int Q, int N>
__device__ __forceinline__ void tc_sum(uint32_t addr, int MT, float (&v)[N]) {
    if constexpr (Q == 1) {
        if constexpr (N == 8) tmem_ld8(addr, v);
        else tmem_ld16(addr, v);
    } else {
        float u[N];
        tc_sum<Q / 2>(addr, MT, v);
        tc_sum<Q / 2>(addr + Q / 2 * MT, MT, u);
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] += u[i];
    }
}
template <int N>
__device__ __forceinline__ void tc_sum_of(int segs, uint32_t addr, int MT, float (&v)[N]) {
    if (segs == 1) tc_sum<1>(addr, MT, v);
    else if (segs == 2) tc_sum<2>(addr, MT, v);
    else tc_sum<4>(addr, MT, v);
}
// f(first column, eight sums) for columns [c0, c1) in eights, read from tensor memory one by one or, with BATCH 16, two at a time: the
// way from there is paid less often, but 16 registers more leave less room beside for the next kernels' CTAs.
template <int BATCH, class F>
__device__ __forceinline__ void tc_columns(int segs, uint32_t addr, int MT, int c0, int c1, F f) {
    auto batch = [&](auto size) {
        constexpr int N = decltype(size)::value;
        float v[N];
        tc_sum_of(segs, addr + c0, MT, v);
#pragma unroll
        for (int i = 0; i < N; i += 8) {
            const float v8[8] = {v[i], v[i + 1], v[i + 2], v[i + 3], v[i + 4], v[i + 5], v[i + 6], v[i + 7]};
            f(c0 + i, v8);
        }
        c0 += N;
    };
    if constexpr (BATCH == 16) {
#pragma unroll 1
        while (c0 + 16 <= c1) batch(std::integral_constant<int, 16>{});
    }
#pragma unroll 1
    while (c0 < c1) batch(std::integral_constant<int, 8>{});
}
// The same over the mailbox's Q sources.
template <int Q>
__device__ __forceinline__ void tc_mail_sum(const float* mail, int src_stride, int row_stride, float (&v)[8]) {
    if constexpr (Q == 1) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = mail[i * row_stride];
    } else {
        float u[8];
        tc_mail_sum<Q / 2>(mail, src_stride, row_stride, v);
        tc_mail_sum<Q / 2>(mail + Q / 2 * src_stride, src_stride, row_stride, u);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] += u[i];
    }
}

template <class Epi, int BATCH>
__global__ void __launch_bounds__(TC_THREADS, 1)
k_gemm_tc(const __grid_constant__ CUtensorMap mapA0, const __grid_constant__ CUtensorMap mapA1,
          const __grid_constant__ CUtensorMap mapX, TcArgs a, Epi ep_all) {
    extern __shared__ unsigned char smem_dyn[];
    __shared__ uint64_t bar_full[TC_MAX_STAGES], bar_empty[TC_MAX_STAGES], bar_done, bar_mail;
    __shared__ uint32_t s_tmem;
    __shared__ int s_bad;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int S = a.splits, rank = blockIdx.x, tile = blockIdx.y;   // the CTAs of one tile are a cluster
    const int m_base = blockIdx.z * a.MT;             // first activation row of this CTA's block
    const int Mb = min(a.MT, a.M - m_base);           // rows of the block
    const Epi ep = ep_all.shifted(m_base);
    tc_stamp(a, 0);
    const int stages = a.stages;
    const uint32_t a_bytes = TC_TILE_N * TC_KCHUNK * 2, stage_bytes = a_bytes + (uint32_t)a.MT * TC_KCHUNK * 2;
    unsigned char* base = smem_dyn + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u);
    const int rpc = TC_TILE_N / S;                    // tile rows this CTA finishes: [rank * rpc, (rank + 1) * rpc)
    float* mail = reinterpret_cast<float*>(base + (size_t)stages * stage_bytes);         // [source][MT][rpc] (S > 1)
    unsigned char* es = reinterpret_cast<unsigned char*>(mail) + (S > 1 ? (size_t)TC_TILE_N * a.MT * 4 : 0);  // epilogue staging
    const int groups = (Mb + 7) / 8;                  // groups of eight activation rows

    if (tid == 0) {
        for (int s = 0; s < stages; ++s) { mbar_init(&bar_full[s], 1); mbar_init(&bar_empty[s], 1); }
        mbar_init(&bar_done, 1);
        mbar_init(&bar_mail, 1);
        s_bad = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        const bool first = blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0;
        if (S > 1) mbar_expect_tx(&bar_mail, (uint32_t)(S * groups * 8 * rpc * 4 + (first ? a.withhold * 4 : 0)));
    }
    const int tmem_cols = a.MT * a.segs < 32 ? 32 : a.MT * a.segs;
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                     "r"(tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    if (S > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");   // waited for before the first push
    tc_stamp(a, 1);
    // Only now may the next kernel's CTAs become resident: every CTA of this grid already owns its
    // tensor-memory columns, so early dependents can never starve it of them.
    pdl_trigger();

    const int k_first = rank * a.chunks / S, n_chunks = (rank + 1) * a.chunks / S - k_first;
    if (warp == 0) {
        if (tc_elect()) {
            // ---- TMA producer.  Weights for the first ring pass go out before the dependency wait.
            auto weights = [&](int c, int s) {
                unsigned char* st = base + (size_t)s * stage_bytes;
                const int x = (k_first + c) * TC_KCHUNK;
                mbar_expect_tx(&bar_full[s], stage_bytes);
                if constexpr (Epi::PAIRED) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        tma_load_2d(st + i * 4096, &mapA0, x, a.row_off + tile * 64 + i * 16, &bar_full[s]);
                        tma_load_2d(st + i * 4096 + 2048, &mapA1, x, a.row_off + tile * 64 + i * 16, &bar_full[s]);
                    }
                } else {
                    tma_load_2d(st, &mapA0, x, a.row_off + tile * TC_TILE_N, &bar_full[s]);
                    tma_load_2d(st + a_bytes / 2, &mapA0, x, a.row_off + tile * TC_TILE_N + 64, &bar_full[s]);
                }
            };
            auto acts = [&](int c, int s) {
                tma_load_2d(base + (size_t)s * stage_bytes + a_bytes, &mapX, (k_first + c) * TC_KCHUNK, m_base, &bar_full[s]);
            };
            for (int c = 0; c < stages; ++c) weights(c, c);
            pdl_wait();
            for (int c = 0; c < stages; ++c) acts(c, c);
            unsigned limit = 4 * a.spin_limit, ph = 0;
            for (int c = stages, s = 0; c < n_chunks; ++c) {
                if (!mbar_wait(&bar_empty[s], ph, limit)) { s_bad = 1; limit = 16; }
                weights(c, s);
                acts(c, s);
                if (++s == stages) { s = 0; ph ^= 1; }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (tc_elect()) {
            // ---- MMA issuer.  The activations come behind the dependency: its wait is not this thread's barriers' to count.
            pdl_wait();
            const uint32_t idesc = tc_idesc(a.MT), d0 = tc_desc(base);
            unsigned limit = 4 * a.spin_limit, ph = 0;
            uint32_t ok = 0;
            for (int c = 0, s = 0, seg = 0, next = 0; c < n_chunks; ++c) {
                const bool first = c == next;   // of a segment: the next accumulator
                if (first) {
                    ++seg;
                    next = (rank * a.segs + seg) * a.chunks / (S * a.segs) - k_first;
                }
                const uint32_t d = tmem + (seg - 1) * a.MT;
                if (!ok && !mbar_wait(&bar_full[s], ph, limit)) { s_bad = 1; limit = 16; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t da = d0 + s * (stage_bytes >> 4), db = da + (a_bytes >> 4);
                uint64_t* const done = &bar_empty[s];
                if (++s == stages) { s = 0; ph ^= 1; }
                if (first) ok = tc_mma4<true, true>(d, da, db, idesc, smem_u32(&bar_full[s]), ph);
                else ok = tc_mma4<false, true>(d, da, db, idesc, smem_u32(&bar_full[s]), ph);
                umma_commit(done);
            }
            umma_commit(&bar_done);
        }
        __syncwarp();
    }
    pdl_wait();
    tc_stamp(a, 2);
    if constexpr (Epi::STAGED) ep.stage(es, tile, Mb, tid);   // while the MMAs run
    // ---- everyone: wait for the accumulator
    const bool done_ok = mbar_wait(&bar_done, 0, 4 * a.spin_limit);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncthreads();
    tc_stamp(a, 3);
    // warps w and w + 4 read tile rows 32 (w & 3) ..: a half of the groups of eight activation rows each
    const int row = (warp & 3) * 32 + lane, split = (groups + 1) / 2 * 8, c0 = warp >> 2 ? split : 0, c1 = warp >> 2 ? groups * 8 : split;
    const uint32_t trow = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    bool mail_ok = true;
    if (S == 1) {
        tc_columns<BATCH>(a.segs, trow, a.MT, c0, c1, [&](int m0, const float (&v)[8]) { tc_apply(ep, tile, row, m0, Mb, v, es); });
    } else {
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");   // every peer has set up its mailbox
        const int owner = row / rpc;
        uint32_t dst, bar;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(smem_u32(mail + (size_t)rank * a.MT * rpc + row % rpc)), "r"(owner));
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(bar) : "r"(smem_u32(&bar_mail)), "r"(owner));
        tc_columns<BATCH>(a.segs, trow, a.MT, c0, c1, [&](int m0, const float (&v)[8]) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
                asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];"
                             ::"r"(dst + (uint32_t)((m0 + j) * rpc * 4)), "f"(v[j]), "r"(bar) : "memory");
        });
        tc_stamp(a, 4);
        {
            const uint32_t addr = smem_u32(&bar_mail);
            mail_ok = false;
            for (unsigned spins = 0; spins < 4 * a.spin_limit && !mail_ok; ++spins) {
                uint32_t ok;
                asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                             : "=r"(ok) : "r"(addr) : "memory");
                mail_ok = ok;
            }
        }
        tc_stamp(a, 5);
        // thread = (row j of the slice, group of eight activation rows); the functors shuffle, and rpc is 32 or 64: warps stay whole
#pragma unroll 1
        for (int e = tid; e < rpc * groups; e += TC_THREADS) {
            const int j = e % rpc, g = e / rpc;
            float v[8];
            const float* box = mail + (size_t)g * 8 * rpc + j;
            if (S == 2) tc_mail_sum<2>(box, a.MT * rpc, rpc, v);
            else tc_mail_sum<4>(box, a.MT * rpc, rpc, v);
            tc_apply(ep, tile, rank * rpc + j, g * 8, Mb, v, es);
        }
    }
    if (!done_ok || !mail_ok || s_bad) {
        // gave up somewhere: what may still be on its way to this CTA's shared memory lands before the CTA retires
        if (lane == 0) atomicOr(a.flag, FLAG_TC_TIMEOUT);
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    }
    tc_stamp(a, 6);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 2) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols) : "memory");
    }
}

// ---------------------------------------------------------------------------
// Row-wise helpers of the batched path.
// ---------------------------------------------------------------------------

// xn[r] = RMSNorm(x[r*row_mul + row_add]) * w   (bf16 rounding as StageNorm)
__global__ void __launch_bounds__(128) k_rmsnorm_rows(const bf16* __restrict__ x, const bf16* __restrict__ w,
                                                      float eps, bf16* __restrict__ out, int K, int row_mul,
                                                      int row_add) {
    pdl_trigger();
    const int r = blockIdx.x;
    __shared__ float red[4];
    const bf16* xr = x + ((size_t)r * row_mul + row_add) * K;
    if (K <= 128 * 8) {
        // one 16-byte piece per thread: the row stays in registers between the two passes and the
        // norm weights (constants) are fetched before the predecessor is waited for
        const int k = threadIdx.x * 8;
        const bool on = k < K;
        const uint4 wv = on ? __ldg(reinterpret_cast<const uint4*>(w + k)) : make_uint4(0, 0, 0, 0);
        pdl_wait();
        float f[8], wf[8], o[8];
        unpack8(on ? __ldcg(reinterpret_cast<const uint4*>(xr + k)) : make_uint4(0, 0, 0, 0), f);
        float ss = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) ss = fmaf(f[j], f[j], ss);
        ss = warp_sum(ss);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
        __syncthreads();
        const float rinv = rsqrtf((red[0] + red[1] + red[2] + red[3]) / (float)K + eps);
        if (on) {
            unpack8(wv, wf);
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] = rbf(f[j] * rinv) * wf[j];
            *reinterpret_cast<uint4*>(out + (size_t)r * K + k) = pack8(o);
        }
        return;
    }
    pdl_wait();
    float ss = 0.f;
    for (int k = threadIdx.x * 8; k < K; k += 128 * 8) {
        float f[8];
        unpack8(__ldcg(reinterpret_cast<const uint4*>(xr + k)), f);
#pragma unroll
        for (int j = 0; j < 8; ++j) ss = fmaf(f[j], f[j], ss);
    }
    ss = warp_sum(ss);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    const float rinv = rsqrtf((red[0] + red[1] + red[2] + red[3]) / (float)K + eps);
    for (int k = threadIdx.x * 8; k < K; k += 128 * 8) {
        float f[8], wf[8], o[8];
        unpack8(__ldcg(reinterpret_cast<const uint4*>(xr + k)), f);
        unpack8(__ldg(reinterpret_cast<const uint4*>(w + k)), wf);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = rbf(f[j] * rinv) * wf[j];
        *reinterpret_cast<uint4*>(out + (size_t)r * K + k) = pack8(o);
    }
}

// Depth-transformer attention for many rows: one CTA per row, one warp per head
// (the same arithmetic as StageRqAttn, written to a buffer instead of a GEMV tile).
template <int K>
__global__ void __launch_bounds__(256) k_rq_attn_rows(StageRqAttn st, bf16* __restrict__ out) {
    pdl_trigger();
    pdl_wait();
    // stage<K>() writes row rr of a tile at Xs + rr*K: aim tile row 0 at this row's output
    st.template stage<K>(out + (size_t)blockIdx.x * K, blockIdx.x, 1);
}

// eos_head for many rows: one warp per row (Linear with bias, model.py:1099).
__global__ void __launch_bounds__(128) k_eos_rows(const bf16* __restrict__ hidden, const bf16* __restrict__ w,
                                                  const bf16* __restrict__ b, bf16* __restrict__ out, int M, int K) {
    pdl_trigger();
    pdl_wait();
    const int r = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (r >= M) return;
    float acc = 0.f;
    for (int k = lane * 8; k < K; k += 256) {
        float x[8], wf[8];
        unpack8(__ldcg(reinterpret_cast<const uint4*>(hidden + (size_t)r * K + k)), x);
        unpack8(__ldg(reinterpret_cast<const uint4*>(w + k)), wf);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc = fmaf(wf[j], x[j], acc);
    }
    acc = warp_sum(acc);
    if (lane == 0) out[r] = f2bf(acc + bf2f(b[0]));
}

}  // namespace vuib
