// The depth transformer's whole codebook loop for several streams in one launch, on the tensor cores.
//
// A thread-block cluster of 8 CTAs owns a group of streams for the whole loop: nothing crosses clusters, so there is no kernel
// hand-over inside it.  CTA c is attention head c, hidden-unit slice c of the MLP and row slice c of each head matrix.  Per layer:
// RMSNorm (replicated) -> its head's q / k / v rows -> its head's attention over its own K / V -> its K-slice of out_proj for all 512
// output rows -> reduce-scatter of the partial rows over the cluster (st.async pushes into the owner's landing zone, summed in
// source order) -> residual add -> all-gather of the new slice; the same for w1 / w3 -> SiLU * gate -> its K-slice of w2.  After a
// position's layers every CTA pushes its logits to the CTA that samples the stream, which pushes the code to all of them.
//
//  * Weights are the M side of tcgen05.mma (128 rows), the group's streams its N side (16 or 32 columns): 40 cycles per 16 of K,
//    which is what reading 128 weight rows from shared memory takes, whatever the number of streams.  One elected thread issues;
//    the eight other warps only see finished tiles in tensor memory.  (Before, the warps that own the streams also ran mma.sync on
//    64 x 64 boxes: ~350 cycles of their instructions a box of 8 KB, 15.8 us a layer.)
//  * The 25.7 MB of layer weights and a 2 MB head per codebook live in L2 and stream through a ring of 32 KB stages, each ONE
//    contiguous bulk copy from a "slot stream" that is laid out once, at binding, in the order of use and in the operand's
//    128-byte-swizzled image.  A producer warp runs ahead through layers, positions and heads.
//  * Each of a layer's 13 tiles has columns of its own in tensor memory, so a tile is never overwritten before the layer is over.
//
// Rounding points are those of the per-launch path (src/vui/model.py:577-635, 908-986); sums are fp32 in another order.  Every wait
// is bounded: a thread whose wait runs out records the device flag and no longer waits.  No load uses cluster multicast.
#pragma once
#include "fused_blocks.cuh"
#include "tc_gemm.cuh"

namespace vuib {

constexpr int DT_CL = 8;                       // CTAs of a cluster
constexpr int DT_CONSUMERS = 256;
constexpr int DT_THREADS = DT_CONSUMERS + 64;  // + producer warp, MMA warp
constexpr int DT_SLOT = 128 * 128;             // a slot: 128 weight rows x 64 bf16
constexpr int DT_STAGE = 2 * DT_SLOT;
constexpr int DT_LAYERS = 4;
constexpr int DT_D = 512;
constexpr int DT_XS = DT_D + 8;                // padded row stride of the residual rows (elements)
constexpr int DT_GROUPS = 15;                  // clusters of 8 that can be resident at once with one CTA per SM
constexpr int DT_HEAD_SLOTS = 16;
constexpr int DT_QKV_SLOTS = 12;               // a layer's first slots: q | k, v

// Slots of a layer and CTA, in order of use: q | k rows of head c per 64 of K (8); v rows, two K-chunks a slot (4); the head's K-slice
// of out_proj per 128 output rows (4); w1 / w3 of 64 hidden units per tile and K-chunk (8 n_ub); the CTA's K-slice of w2 per 128
// output rows and 64 units (4 n_ub).
__host__ __device__ inline int dt_slots_per_layer(int n_ub) { return 16 + 12 * n_ub; }

struct DtStreamBuild {
    const bf16* wqkv[DT_LAYERS]; const bf16* out[DT_LAYERS]; const bf16* w1[DT_LAYERS]; const bf16* w3[DT_LAYERS];
    const bf16* w2[DT_LAYERS];
    const bf16* head;              // ((Q - 1) * CS, 512)
    unsigned char* layers;         // [n_layers][8 CTAs][slots][16384]
    unsigned char* head_out;       // [Q - 1][8 CTAs][16][16384]
    int n_layers, ffn, upc, n_ub, CS, n_head_pos;
};

// One CTA per slot of the stream.
static __global__ void __launch_bounds__(256) k_build_dt_stream(DtStreamBuild b) {
    const int spl = dt_slots_per_layer(b.n_ub), n_layer_slots = b.n_layers * DT_CL * spl;
    int slot = blockIdx.x;
    const bool head = slot >= n_layer_slots;
    unsigned char* dst = head ? b.head_out + (size_t)(slot - n_layer_slots) * DT_SLOT : b.layers + (size_t)slot * DT_SLOT;
    int l = 0, c, j;
    if (head) { slot -= n_layer_slots; l = slot / (DT_CL * DT_HEAD_SLOTS); c = slot / DT_HEAD_SLOTS % DT_CL; j = slot % DT_HEAD_SLOTS; }
    else { l = slot / (DT_CL * spl); c = slot / spl % DT_CL; j = slot % spl; }
    for (int i = threadIdx.x; i < 128 * 8; i += 256) {       // 16-byte pieces: row r, piece q
        const int r = i >> 3, q = i & 7;
        const bf16* src = nullptr;
        if (head) src = b.head + ((size_t)l * b.CS + c * 256 + (j / 8) * 128 + r) * DT_D + (j % 8) * 64 + q * 8;
        else if (j < 8) src = b.wqkv[l] + (size_t)((r / 64) * DT_D + c * HD + r % 64) * DT_D + j * 64 + q * 8;
        else if (j < 12) src = b.wqkv[l] + (size_t)(2 * DT_D + c * HD + r % 64) * DT_D + ((j - 8) * 2 + r / 64) * 64 + q * 8;
        else if (j < 16) src = b.out[l] + (size_t)((j - 12) * 128 + r) * DT_D + c * HD + q * 8;
        else if (j < 16 + 8 * b.n_ub) {
            // a warp's 32 lanes of a tile hold 16 rows of w1 and the same 16 units' rows of w3
            const int t = (j - 16) / 8, kb = (j - 16) % 8, unit = t * 64 + (r / 32) * 16 + (r & 15);
            if (unit < b.upc) src = ((r & 31) < 16 ? b.w1[l] : b.w3[l]) + (size_t)(c * b.upc + unit) * DT_D + kb * 64 + q * 8;
        } else {
            const int t = (j - 16 - 8 * b.n_ub) / b.n_ub, ub = (j - 16 - 8 * b.n_ub) % b.n_ub, unit = ub * 64 + q * 8;
            if (unit < b.upc) src = b.w2[l] + (size_t)(t * 128 + r) * b.ffn + c * b.upc + unit;   // upc is a multiple of 8
        }
        const uint4 v = src ? __ldg(reinterpret_cast<const uint4*>(src)) : make_uint4(0, 0, 0, 0);
        *reinterpret_cast<uint4*>(dst + r * 128 + ((q ^ (r & 7)) << 4)) = v;
    }
}

struct DepthTcArgs {
    const unsigned char* layers;
    const unsigned char* head;
    int slots_per_layer, n_ub;
    int B, r;         // streams in all, streams of a group
    int n_layers;     // <= DT_LAYERS
    int Q, Qn;        // quantizers of the model, codebooks to emit (positions to run)
    int CS;
    int upc;          // hidden units per CTA = rq_ffn / 8 (<= 192)
    int max_rows;     // row stride of the depth K/V scratch
    float eps;
    const bf16* x2;   // (B, 2, 512): tokens of depth positions 0 and 1
    bf16* kc;         // (layers, max_rows, Q, 512)
    bf16* vc;
    const bf16* attn_norm[DT_LAYERS];
    const bf16* mlp_norm[DT_LAYERS];
    const bf16* final_norm;
    bf16* tap;        // optional copy of the logits: row stride (Q-1)*CS, codebook i at +i*CS
    SampleArgs sa;    // everything but the per-position fields
    int32_t* flag;
    unsigned spin_limit;
    unsigned long long* dbg;  // optional: device-clock stamps of CTA 0 at position 8, layer 1 (profiling aid)
};

template <int N, int RMAX, int STAGES>
struct DepthTcSmem {
    alignas(1024) unsigned char ring[STAGES][DT_STAGE];
    alignas(1024) unsigned char h[8][N * 128];          // normed activations, MMA operand: [K / 64][stream][128 bytes, swizzled]
    alignas(1024) unsigned char attn[N * 128];          // this head's attention output, likewise
    alignas(1024) unsigned char g[3][N * 128];          // this CTA's SwiGLU activations, likewise
    alignas(16) bf16 x[RMAX][DT_XS];                    // residual stream of the group's streams (same in every CTA)
    alignas(16) bf16 qkv[3][RMAX][HD];                  // this head's q, new k, new v
    union {     // a position's logits come when its exchanges are over, and the next exchange follows the codes drawn from them
        alignas(16) float land[DT_CL][RMAX][HD];        // reduce-scatter landing zone [source CTA][stream][column]
        alignas(16) bf16 logits[(RMAX + 7) / 8][2048];  // of the streams that this CTA samples
    };
    alignas(16) bf16 norm_w[2 * DT_LAYERS + 1][DT_D];   // attention and MLP norms of the layers in turn, final norm
    int codes[RMAX];
    SampleKey keys[(RMAX + 7) / 8];                     // of the streams that this CTA samples
    alignas(8) uint64_t full[STAGES], empty[STAGES];
    uint64_t h_ready, attn_ready, g_ready;              // consumers -> MMA thread
    uint64_t d_qk, d_v, d_out[4], d_g[3], d_w2[4], d_head[2];   // finished tiles
    uint64_t bar_rs, bar_ag, bar_logits, bar_codes;
    uint32_t tmem;
    SampleSmem samp;
};

__device__ __forceinline__ void dt_bar() { bar_named(1, DT_CONSUMERS); }

// A thread's bounded waits: after the first that runs out it only looks once.
struct DtWait {
    int32_t* flag;
    unsigned limit;
    __device__ __forceinline__ void local(uint64_t* bar, unsigned parity) {
        if (!mbar_wait(bar, parity, limit)) expired();
    }
    __device__ __forceinline__ void cluster(uint64_t* bar, unsigned parity) {   // what peers pushed: cluster-scope acquire
        const uint32_t a = smem_u32(bar);
        for (unsigned spins = 0; spins < limit; ++spins) {
            uint32_t ok;
            asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                         : "=r"(ok) : "r"(a), "r"(parity) : "memory");
            if (ok) return;
        }
        expired();
    }
    __device__ __forceinline__ void expired() {
        if (limit > 1) atomicOr(flag, FLAG_COPY_TIMEOUT);
        limit = 1;
    }
    // A CTA that gave up a wait must not retire with copies or pushes on their way to its shared memory; the launch takes 2 ms at most.
    __device__ __forceinline__ void linger() const {
        if (limit == 1)
            for (int i = 0; i < 1000; ++i) __nanosleep(10000);
    }
};

__device__ __forceinline__ void dt_push_b32(uint32_t dst, uint32_t bar, uint32_t v) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(dst), "r"(v), "r"(bar) : "memory");
}
template <int N, bool FIRST, bool TEST>
__device__ __forceinline__ uint32_t dt_mma4(uint32_t d, uint32_t a, uint32_t b, uint32_t bar, uint32_t parity) {
    return tc_mma4<FIRST, TEST>(d, a, b, tc_idesc(N), bar, parity);
}

// The first columns of this thread's row of a tile: as many as hold RMAX streams.
template <int RMAX>
constexpr int DT_COLS = RMAX <= 8 ? 8 : RMAX <= 16 ? 16 : 32;
template <int K>
__device__ __forceinline__ void dt_tile(uint32_t addr, float (&v)[K]) {
    static_assert(K == 8 || K == 16 || K == 32, "columns");
    if constexpr (K == 32) tmem_ld32(addr, v);
    else if constexpr (K == 16) tmem_ld16(addr, v);
    else tmem_ld8(addr, v);
}

// RMSNorm of the residual rows into the MMA operand h: warp w takes streams w, w + 8, ...
template <class S>
__device__ __forceinline__ void dt_norm(S& sm, const bf16* w, float eps, int nv) {   // w in shared memory
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float w0[8], w1[8];
    unpack8(*reinterpret_cast<const uint4*>(w + lane * 16), w0);
    unpack8(*reinterpret_cast<const uint4*>(w + lane * 16 + 8), w1);
    for (int n = warp; n < nv; n += DT_CONSUMERS / 32) {
        float v0[8], v1[8];
        unpack8(*reinterpret_cast<const uint4*>(&sm.x[n][lane * 16]), v0);
        unpack8(*reinterpret_cast<const uint4*>(&sm.x[n][lane * 16 + 8]), v1);
        float ss = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) ss = fmaf(v0[j], v0[j], ss);
#pragma unroll
        for (int j = 0; j < 8; ++j) ss = fmaf(v1[j], v1[j], ss);
        ss = warp_sum(ss);
        const float rinv = rsqrtf(ss / (float)DT_D + eps);
        float o0[8], o1[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) { o0[j] = rbf(v0[j] * rinv) * w0[j]; o1[j] = rbf(v1[j] * rinv) * w1[j]; }
        unsigned char* row = sm.h[lane >> 2] + n * 128;
        const int q = (lane & 3) * 2;
        *reinterpret_cast<uint4*>(row + ((q ^ (n & 7)) << 4)) = pack8(o0);
        *reinterpret_cast<uint4*>(row + (((q + 1) ^ (n & 7)) << 4)) = pack8(o1);
    }
}

// What this warp wrote to an MMA operand (and read from tensor memory) is done: one arrival of eight.
__device__ __forceinline__ void dt_publish(uint64_t* bar) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    if ((threadIdx.x & 31) == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void dt_wait_tile(DtWait& w, uint64_t* bar, unsigned parity) {
    w.local(bar, parity);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncwarp();
}

// The four 128-row tiles of a column-split product: a thread's row goes to the CTA that owns its column.  The lanes of a warp are 32
// neighbouring columns, so that a push is one run of 128 bytes on the way to the peer (with a run of streams per lane, or a stream
// per lane in the sum below, an exchange took 0.8 us longer).
template <int N, int RMAX, class S>
__device__ __forceinline__ void dt_push_partials(S& sm, DtWait& w, uint64_t* done, unsigned parity, uint32_t tmem, int c, int nv) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quarter = warp & 3, half = warp >> 2;
    for (int t = half; t < 4; t += 2) {
        const int owner = t * 2 + (quarter >> 1), col = (quarter & 1) * 32 + lane;
        const uint32_t dst = peer_addr(&sm.land[c][0][col], owner), bar = peer_addr(&sm.bar_rs, owner);
        dt_wait_tile(w, &done[t], parity);
        float v[DT_COLS<RMAX>];
        dt_tile(tmem + ((uint32_t)(quarter * 32) << 16) + t * N, v);
#pragma unroll
        for (int n = 0; n < RMAX; ++n)
            if (n < nv) push_f32(dst + n * (HD * 4), bar, v[n]);
    }
}

// Once all eight sources have landed, the owner adds them in source order to its slice of the residual and sends the new slice to
// every CTA's copy of x.  An item is two columns of a stream.
template <int RMAX, class S>
__device__ __forceinline__ void dt_residual_exchange(S& sm, DtWait& w, int c, unsigned& phase, int nv, const uint32_t (&peer)[DT_CL]) {
    const int tid = threadIdx.x;
    w.cluster(&sm.bar_rs, phase & 1);
    for (int e = tid; e < nv * (HD / 2); e += DT_CONSUMERS) {
        const int n = e / (HD / 2), col = (e % (HD / 2)) * 2;
        float2 p[DT_CL];
#pragma unroll
        for (int src = 0; src < DT_CL; ++src) p[src] = *reinterpret_cast<const float2*>(&sm.land[src][n][col]);
        float s0 = 0.f, s1 = 0.f;
#pragma unroll
        for (int src = 0; src < DT_CL; ++src) { s0 += p[src].x; s1 += p[src].y; }
        const __nv_bfloat162 old = *reinterpret_cast<const __nv_bfloat162*>(&sm.x[n][c * HD + col]);
        const __nv_bfloat162 now = __floats2bfloat162_rn(__low2float(old) + rbf(s0), __high2float(old) + rbf(s1));
        const uint32_t bits = *reinterpret_cast<const uint32_t*>(&now);
        const uint32_t off = smem_u32(&sm.x[n][c * HD + col]) - smem_u32(&sm), bar = smem_u32(&sm.bar_ag) - smem_u32(&sm);
#pragma unroll
        for (int q = 0; q < DT_CL; ++q) dt_push_b32(peer[q] + off, peer[q] + bar, bits);
    }
    if (tid == 0) mbar_expect_tx(&sm.bar_rs, (uint32_t)(DT_CL * HD * nv * 4));  // armed for the next round
    w.cluster(&sm.bar_ag, phase & 1);
    if (tid == 0) mbar_expect_tx(&sm.bar_ag, (uint32_t)(DT_CL * nv * HD * 2));
    ++phase;
}

template <int N, int RMAX, int STAGES>
__global__ void __launch_bounds__(DT_THREADS, 1) k_depth_tc(const __grid_constant__ DepthTcArgs a) {
    using S = DepthTcSmem<N, RMAX, STAGES>;
    extern __shared__ __align__(1024) unsigned char dt_smem[];
    S& sm = *reinterpret_cast<S*>(dt_smem);
    const int c = blockIdx.x % DT_CL;                  // head / slice of this CTA
    const int b0 = (blockIdx.x / DT_CL) * a.r;         // first stream of the group
    const int nv = min(a.r, a.B - b0);                 // its streams
    const int mine = (nv - c + DT_CL - 1) / DT_CL;     // streams this CTA samples (may be 0)
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n_pos = a.Qn, n_ub = a.n_ub;             // depth positions 0 .. Qn - 1; position p >= 1 yields codebook p
    // Position 0 yields no codebook: of its last layer the others need the keys and values alone (12 frames of 256 streams 41.96 -> 41.66
    // ms; of 16 and 64 streams the same as before).
    const auto keys_only = [&](int pos, int l) { return pos == 0 && l == a.n_layers - 1; };
    if (tid == 0) {
        for (int i = 0; i < STAGES; ++i) { mbar_init(&sm.full[i], 1); mbar_init(&sm.empty[i], 1); }
        mbar_init(&sm.h_ready, DT_CONSUMERS / 32);
        mbar_init(&sm.attn_ready, DT_CONSUMERS / 32);
        mbar_init(&sm.g_ready, DT_CONSUMERS / 32);
        mbar_init(&sm.d_qk, 1);
        mbar_init(&sm.d_v, 1);
        for (int i = 0; i < 4; ++i) { mbar_init(&sm.d_out[i], 1); mbar_init(&sm.d_w2[i], 1); }
        for (int i = 0; i < 3; ++i) mbar_init(&sm.d_g[i], 1);
        for (int i = 0; i < 2; ++i) mbar_init(&sm.d_head[i], 1);
        mbar_init(&sm.bar_rs, 1);
        mbar_init(&sm.bar_ag, 1);
        mbar_init(&sm.bar_logits, 1);
        mbar_init(&sm.bar_codes, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_expect_tx(&sm.bar_rs, (uint32_t)(DT_CL * HD * nv * 4));
        mbar_expect_tx(&sm.bar_ag, (uint32_t)(DT_CL * nv * HD * 2));
        if (mine > 0) mbar_expect_tx(&sm.bar_logits, (uint32_t)(mine * 2048 * 2));
        mbar_expect_tx(&sm.bar_codes, (uint32_t)(nv * 4));
    }
    if (warp == DT_CONSUMERS / 32 + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = sm.tmem;
    pdl_trigger();     // every CTA owns its tensor memory by now
    cluster_arrive();
    // columns of a layer's tiles
    const uint32_t t_qk = tmem, t_v = tmem + N, t_out = tmem + 2 * N, t_g = tmem + 6 * N, t_w2 = tmem + 9 * N, t_head = tmem + 13 * N;

    if (warp == DT_CONSUMERS / 32) {
        // ---------------------------------------------------------------- producer: the slot stream, stage by stage
        if (tc_elect()) {
            DtWait w{a.flag, 16u * a.spin_limit};
            int st = 0;
            unsigned ph = 1;
            bool waited = false;
            bool filled = false;
            auto stages = [&](const unsigned char* src, int n) {
                for (int i = 0; i < n; ++i) {
                    if (filled) {
                        if (!waited) { pdl_wait(); waited = true; }   // the ring is full until the dependency is met
                        w.local(&sm.empty[st], ph);
                    }
                    mbar_expect_tx(&sm.full[st], DT_STAGE);
                    bulk_g2s(sm.ring[st], src + (size_t)i * DT_STAGE, DT_STAGE, &sm.full[st]);
                    if (++st == STAGES) { st = 0; ph ^= 1; filled = true; }
                }
            };
            for (int pos = 0; pos < n_pos; ++pos) {
                for (int l = 0; l < a.n_layers; ++l)
                    stages(a.layers + (size_t)(l * DT_CL + c) * a.slots_per_layer * DT_SLOT, keys_only(pos, l) ? DT_QKV_SLOTS / 2 : a.slots_per_layer / 2);
                if (pos >= 1) stages(a.head + (size_t)((pos - 1) * DT_CL + c) * DT_HEAD_SLOTS * DT_SLOT, DT_HEAD_SLOTS / 2);
            }
            w.linger();
        }
        __syncwarp();
        cluster_wait();
    } else if (warp == DT_CONSUMERS / 32 + 1) {
        // ---------------------------------------------------------------- MMA thread
        if (tc_elect()) {
            pdl_wait();   // its length is not this thread's barriers' to count
            DtWait w{a.flag, 16u * a.spin_limit};
            int st = 0;
            unsigned ph = 0, ph_h = 0, ph_l = 0;
            uint32_t ok = 0;
            const uint32_t ring0 = tc_desc(sm.ring[0]), h0 = tc_desc(sm.h[0]), at0 = tc_desc(sm.attn), g0 = tc_desc(sm.g[0]);
            constexpr uint32_t CHUNK = N * 128 >> 4, SLOT = DT_SLOT >> 4;
            uint32_t slot = 0, nbar = 0, nph = 0;
            // the stage's first slot; where the next stage will be
            auto open = [&] {
                if (!ok) w.local(&sm.full[st], ph);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                slot = ring0 + st * (DT_STAGE >> 4);
                const int n1 = st + 1 == STAGES ? 0 : st + 1;
                nbar = smem_u32(&sm.full[n1]);
                nph = n1 ? ph : ph ^ 1;
            };
            auto close = [&] {
                umma_commit(&sm.empty[st]);
                if (++st == STAGES) { st = 0; ph ^= 1; }
            };
            auto need = [&](uint64_t* bar, unsigned parity) {
                w.local(bar, parity);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            };
            // eight K-chunks of h for one tile
            auto tile8 = [&](uint32_t d) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    open();
                    if (i == 0) dt_mma4<N, true, false>(d, slot, h0, 0, 0);
                    else dt_mma4<N, false, false>(d, slot, h0 + 2 * i * CHUNK, 0, 0);
                    ok = dt_mma4<N, false, true>(d, slot + SLOT, h0 + (2 * i + 1) * CHUNK, nbar, nph);
                    close();
                }
            };
            for (int pos = 0; pos < n_pos; ++pos) {
                for (int l = 0; l < a.n_layers; ++l) {
                    need(&sm.h_ready, ph_h);
                    ph_h ^= 1;
                    tile8(t_qk);
                    umma_commit(&sm.d_qk);
#pragma unroll
                    for (int i = 0; i < 2; ++i) {   // v: 64 rows a chunk; the other 64 rows of the tile are not looked at
                        open();
                        if (i == 0) dt_mma4<N, true, false>(t_v, slot, h0, 0, 0);
                        else dt_mma4<N, false, false>(t_v, slot, h0 + 4 * CHUNK, 0, 0);
                        dt_mma4<N, false, false>(t_v, slot + SLOT / 2, h0 + (4 * i + 1) * CHUNK, 0, 0);
                        dt_mma4<N, false, false>(t_v, slot + SLOT, h0 + (4 * i + 2) * CHUNK, 0, 0);
                        ok = dt_mma4<N, false, true>(t_v, slot + SLOT / 2 * 3, h0 + (4 * i + 3) * CHUNK, nbar, nph);
                        close();
                    }
                    umma_commit(&sm.d_v);
                    if (keys_only(pos, l)) break;
                    need(&sm.attn_ready, ph_l);
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        open();
                        dt_mma4<N, true, false>(t_out + 2 * i * N, slot, at0, 0, 0);
                        umma_commit(&sm.d_out[2 * i]);
                        ok = dt_mma4<N, true, true>(t_out + (2 * i + 1) * N, slot + SLOT, at0, nbar, nph);
                        umma_commit(&sm.d_out[2 * i + 1]);
                        close();
                    }
                    need(&sm.h_ready, ph_h);
                    ph_h ^= 1;
                    for (int t = 0; t < n_ub; ++t) {
                        tile8(t_g + t * N);
                        umma_commit(&sm.d_g[t]);
                    }
                    need(&sm.g_ready, ph_l);
                    for (int s = 0, t = 0, ub = 0; s < 4 * n_ub; s += 2) {
                        open();
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const uint32_t d = t_w2 + t * N, b = g0 + ub * CHUNK, x = slot + i * SLOT;
                            if (i == 0) { if (ub == 0) dt_mma4<N, true, false>(d, x, b, 0, 0); else dt_mma4<N, false, false>(d, x, b, 0, 0); }
                            else { if (ub == 0) ok = dt_mma4<N, true, true>(d, x, b, nbar, nph); else ok = dt_mma4<N, false, true>(d, x, b, nbar, nph); }
                            if (++ub == n_ub) {
                                umma_commit(&sm.d_w2[t]);
                                ub = 0;
                                ++t;
                            }
                        }
                        close();
                    }
                    ph_l ^= 1;
                }
                if (pos == 0) continue;
                need(&sm.h_ready, ph_h);
                ph_h ^= 1;
                for (int t = 0; t < 2; ++t) {
                    tile8(t_head + t * N);
                    umma_commit(&sm.d_head[t]);
                }
            }
            w.linger();
        }
        __syncwarp();
        cluster_wait();
    } else {
        // ---------------------------------------------------------------- consumers
        pdl_wait();
        cluster_wait();
        DtWait w{a.flag, a.spin_limit};
        // What the loop needs of global memory is fetched here, or long before it is used: a small load queues up behind the
        // ring's copies on their way to the SM, 1 to 2 us.
        for (int i = tid; i < (2 * DT_LAYERS + 1) * (DT_D / 8); i += DT_CONSUMERS) {
            const int r = i / (DT_D / 8), l = min(r / 2, a.n_layers - 1);
            const bf16* src = r == 2 * DT_LAYERS ? a.final_norm : r & 1 ? a.mlp_norm[l] : a.attn_norm[l];
            *reinterpret_cast<uint4*>(&sm.norm_w[r][(i % (DT_D / 8)) * 8]) = __ldg(reinterpret_cast<const uint4*>(src) + i % (DT_D / 8));
        }
        if (tid < RMAX) sm.codes[tid] = 0;   // an index also where the wait for the codes runs out
        if (tid < mine) sm.keys[tid] = sample_key(a.sa, b0 + c + tid * DT_CL, true);   // read behind many barriers
        const int quarter = warp & 3, half = warp >> 2;
        const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
        unsigned phase = 0, ph_q = 0, ph_l = 0, ph_pos = 0;   // parities of the q/k/v tiles and of a layer's others
        uint32_t peer[DT_CL];   // this CTA's shared memory at every CTA of the cluster
#pragma unroll
        for (int q = 0; q < DT_CL; ++q) peer[q] = peer_addr(&sm, q);
        dt_bar();
        // earlier keys and values of this warp's first SETS streams, a layer ahead in registers
        constexpr int SETS = RMAX > 8 ? 2 : 1;
        const int s8 = lane & 7, g4 = lane >> 3;
        uint4 kr[SETS][4], vr[SETS][4];
        auto fetch = [&](uint4 (&k4)[4], uint4 (&v4)[4], int l, int n, int n_keys) {
            const size_t row = ((size_t)l * a.max_rows + b0 + n) * a.Q * DT_D + c * HD + s8 * 8;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int tk = u * 4 + g4;
                const bool ok = tk < n_keys;
                k4[u] = v4[u] = make_uint4(0, 0, 0, 0);
                if (ok) {
                    k4[u] = ld_l2(a.kc + row + (size_t)tk * DT_D);
                    v4[u] = ld_l2(a.vc + row + (size_t)tk * DT_D);
                }
            }
        };
#pragma unroll
        for (int i = 0; i < SETS; ++i)
#pragma unroll
            for (int u = 0; u < 4; ++u) kr[i][u] = vr[i][u] = make_uint4(0, 0, 0, 0);   // position 0 has no earlier keys
        for (int pos = 0; pos < n_pos; ++pos) {
            // ---- the position's token rows; a warp normalises the rows that it fetches
            if (pos >= 2) {
                w.cluster(&sm.bar_codes, pos & 1);
                if (tid == 0) mbar_expect_tx(&sm.bar_codes, (uint32_t)(nv * 4));
            }
            for (int n = warp; n < nv; n += DT_CONSUMERS / 32) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int k = lane * 16 + i * 8;
                    if (pos < 2) {
                        *reinterpret_cast<uint4*>(&sm.x[n][k]) = __ldcg(reinterpret_cast<const uint4*>(a.x2 + ((size_t)(b0 + n) * 2 + pos) * DT_D + k));
                    } else {
                        float e[8], p[8];
                        unpack8(__ldg(reinterpret_cast<const uint4*>(a.sa.code_emb + ((size_t)(pos - 1) * a.CS + sm.codes[n]) * DT_D + k)), e);
                        unpack8(__ldg(reinterpret_cast<const uint4*>(a.sa.pos_emb + (size_t)pos * DT_D + k)), p);
#pragma unroll
                        for (int j = 0; j < 8; ++j) e[j] += p[j];
                        *reinterpret_cast<uint4*>(&sm.x[n][k]) = pack8(e);
                    }
                }
            }
            __syncwarp();
            for (int l = 0; l < a.n_layers; ++l, ph_q ^= 1) {
                bf16* kcl = a.kc + (size_t)l * a.max_rows * a.Q * DT_D;
                bf16* vcl = a.vc + (size_t)l * a.max_rows * a.Q * DT_D;
                unsigned long long* dbg = (pos == 8 && l == 1) ? a.dbg : nullptr;
                fb_stamp(dbg, 0);
                dt_norm(sm, sm.norm_w[2 * l], a.eps, nv);
                dt_publish(&sm.h_ready);
                fb_stamp(dbg, 1);
                // ---- q and k rows to warps 0-3, v rows to warps 4 and 5
                dt_wait_tile(w, half ? &sm.d_v : &sm.d_qk, ph_q);
                if (half == 0 || quarter < 2) {
                    float v[DT_COLS<RMAX>];
                    dt_tile((half ? t_v : t_qk) + lanes, v);
                    const int which = half ? 2 : quarter >> 1, dim = (quarter & 1) * 32 + lane;
                    bf16* cache = which == 1 ? kcl : vcl;
#pragma unroll
                    for (int n = 0; n < RMAX; ++n)
                        if (n < nv) {
                            const bf16 o = f2bf(v[n]);
                            sm.qkv[which][n][dim] = o;
                            if (which > 0) cache[((size_t)(b0 + n) * a.Q + pos) * DT_D + c * HD + dim] = o;
                        }
                }
                dt_bar();
                fb_stamp(dbg, 2);
                auto fetch_next = [&] {   // the next layer's keys and values, or the next position's first layer's
                    const bool wrap = l == a.n_layers - 1;
#pragma unroll
                    for (int i = 0; i < SETS; ++i)
                        if (warp + 8 * i < nv) fetch(kr[i], vr[i], wrap ? 0 : l + 1, warp + 8 * i, wrap ? pos + 1 : pos);
                };
                if (keys_only(pos, l)) {
                    fetch_next();
                    continue;
                }
                // ---- attention of head c: one warp per stream, keys [0, pos) + the new key
                auto attend = [&](int n, const uint4 (&k4)[4], const uint4 (&v4)[4]) {
                    // Group g4 of eight lanes has keys g4, g4 + 4, .. and lane s8 of it eight of the 64 dimensions; the new key is every
                    // group's fifth, counted once.  All scores first, one maximum, one exponential a key: with a running softmax
                    // (each key waiting for the one before) the 15 keys of the last position took three times as long.
                    float qf[8], t8[8], sc[5];
                    unpack8(*reinterpret_cast<const uint4*>(&sm.qkv[0][n][s8 * 8]), qf);
#pragma unroll
                    for (int u = 0; u < 5; ++u) {
                        unpack8(u < 4 ? k4[u < 4 ? u : 0] : *reinterpret_cast<const uint4*>(&sm.qkv[1][n][s8 * 8]), t8);
                        sc[u] = 0.f;
#pragma unroll
                        for (int j = 0; j < 8; ++j) sc[u] = fmaf(qf[j], t8[j], sc[u]);
                    }
#pragma unroll
                    for (int o = 1; o <= 4; o <<= 1)
#pragma unroll
                        for (int u = 0; u < 5; ++u) sc[u] += __shfl_xor_sync(0xffffffffu, sc[u], o);
                    float m = sc[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) if (u * 4 + g4 < pos) m = fmaxf(m, sc[u]);
                    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 8));
                    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 16));
                    float lsum = 0.f, acc8[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc8[j] = 0.f;
#pragma unroll
                    for (int u = 0; u < 5; ++u) {
                        unpack8(u < 4 ? v4[u < 4 ? u : 0] : *reinterpret_cast<const uint4*>(&sm.qkv[2][n][s8 * 8]), t8);
                        const bool on = u < 4 ? u * 4 + g4 < pos : g4 == 0;
                        const float p = on ? __expf((sc[u] - m) * 0.125f) : 0.f;
                        lsum += p;
#pragma unroll
                        for (int j = 0; j < 8; ++j) acc8[j] = fmaf(p, t8[j], acc8[j]);
                    }
#pragma unroll
                    for (int o = 8; o <= 16; o <<= 1) {
                        lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
#pragma unroll
                        for (int j = 0; j < 8; ++j) acc8[j] += __shfl_xor_sync(0xffffffffu, acc8[j], o);
                    }
                    if (g4 == 0) {
                        const float inv = 1.f / lsum;
#pragma unroll
                        for (int j = 0; j < 8; ++j) acc8[j] *= inv;
                        *reinterpret_cast<uint4*>(sm.attn + n * 128 + ((s8 ^ (n & 7)) << 4)) = pack8(acc8);
                    }
                };
#pragma unroll
                for (int i = 0; i < SETS; ++i)
                    if (warp + 8 * i < nv) attend(warp + 8 * i, kr[i], vr[i]);
                for (int n = warp + 8 * SETS; n < nv; n += 8) {   // 17 and 18 streams: the last two are fetched when they are needed
                    uint4 k4[4], v4[4];
                    fetch(k4, v4, l, n, pos);
                    attend(n, k4, v4);
                }
                dt_publish(&sm.attn_ready);
                fetch_next();
                fb_stamp(dbg, 3);
                dt_push_partials<N, RMAX>(sm, w, sm.d_out, ph_l, t_out, c, nv);
                fb_stamp(dbg, 4);
                dt_residual_exchange<RMAX>(sm, w, c, phase, nv, peer);
                fb_stamp(dbg, 5);
                // ---- MLP: this CTA's hidden units
                dt_norm(sm, sm.norm_w[2 * l + 1], a.eps, nv);
                dt_publish(&sm.h_ready);
                fb_stamp(dbg, 6);
                // lanes l and l + 16 hold w1 and w3 sums of one unit: the lower one gates the first half of the streams.  The last tile
                // of three, which nothing follows, is shared by the two halves of the warps.
                for (int t = half; t < n_ub; t += t == 0 && half == 0 ? 2 : 1) {
                    const bool shared = t == 2;
                    dt_wait_tile(w, &sm.d_g[t], ph_l);
                    constexpr int HN = (RMAX + 1) / 2;
                    float v[DT_COLS<RMAX>];
                    dt_tile(t_g + t * N + lanes, v);
                    const bool low = lane < 16;
                    const int u = quarter * 16 + (lane & 15);
#pragma unroll
                    for (int i = 0; i < HN; ++i) {
                        if (shared && (i & 1) != half) continue;
                        const float got = __shfl_xor_sync(0xffffffffu, low ? v[i + HN] : v[i], 16);
                        const float a1 = rbf(low ? v[i] : got), a3 = rbf(low ? got : v[i + HN]);
                        const float sl = rbf(silu(a1));
                        const int n = low ? i : i + HN;
                        *reinterpret_cast<bf16*>(sm.g[t] + n * 128 + (((u >> 3) ^ (n & 7)) << 4) + (u & 7) * 2) = f2bf(sl * a3);
                    }
                }
                dt_publish(&sm.g_ready);
                fb_stamp(dbg, 7);
                dt_push_partials<N, RMAX>(sm, w, sm.d_w2, ph_l, t_w2, c, nv);
                fb_stamp(dbg, 8);
                dt_residual_exchange<RMAX>(sm, w, c, phase, nv, peer);
                fb_stamp(dbg, 9);
                ph_l ^= 1;
            }
            if (pos == 0) continue;
            unsigned long long* dbg = pos == 8 ? a.dbg : nullptr;
            // ---- head of codebook `pos`: this CTA's 256 rows to the CTAs that sample the streams
            dt_norm(sm, sm.norm_w[2 * DT_LAYERS], a.eps, nv);
            dt_publish(&sm.h_ready);
            fb_stamp(dbg, 10);
            dt_wait_tile(w, &sm.d_head[half], ph_pos);
            {
                constexpr int K = DT_COLS<RMAX>;
                float v[K];
                dt_tile(t_head + half * N + lanes, v);
                const int row = c * 256 + half * 128 + quarter * 32 + lane;
#pragma unroll
                for (int n = 0; n < RMAX; n += 2) {
                    if (n >= nv) break;
                    const float v1 = v[n + 1];   // RMAX is even
                    const bool odd = lane & 1;
                    const float got = __shfl_xor_sync(0xffffffffu, odd ? v[n] : v1, 1);
                    const __nv_bfloat162 pair = odd ? __floats2bfloat162_rn(got, v1) : __floats2bfloat162_rn(v[n], got);
                    const int s = n + odd;
                    if (s < nv)
                        dt_push_b32(peer_addr(&sm.logits[s / DT_CL][row & ~1], s % DT_CL), peer_addr(&sm.bar_logits, s % DT_CL),
                                    *reinterpret_cast<const uint32_t*>(&pair));
                    if (a.tap) {
                        bf16* t0 = a.tap + (size_t)(b0 + n) * (a.Q - 1) * a.CS + (size_t)(pos - 1) * a.CS + row;
                        t0[0] = f2bf(v[n]);
                        if (n + 1 < nv) t0[(size_t)(a.Q - 1) * a.CS] = f2bf(v1);
                    }
                }
            }
            fb_stamp(dbg, 11);
            const float u_first = mine > 0 ? sample_uniform(sm.keys[0], pos) : 0.f;   // while the logits are on their way
            if (mine > 0) {
                w.cluster(&sm.bar_logits, ph_pos);
                if (tid == 0) mbar_expect_tx(&sm.bar_logits, (uint32_t)(mine * 2048 * 2));
            }
            ph_pos ^= 1;
            fb_stamp(dbg, 12);
            for (int i = 0; i < mine; ++i) {
                const int n = c + i * DT_CL;
                const SampleKey key = sm.keys[i];
                const uint4 raw = *reinterpret_cast<const uint4*>(&sm.logits[i][tid * SAMPLE_EL]);
                const int code = sample_rq(raw, key, i == 0 ? u_first : sample_uniform(key, pos), tid, sm.samp, 1);
                // the last position's peers may already have retired: nothing is sent to them
                if (tid < DT_CL && pos + 1 < n_pos) dt_push_b32(peer_addr(&sm.codes[n], tid), peer_addr(&sm.bar_codes, tid), (uint32_t)code);
                if (tid == DT_CL) {
                    a.sa.code_cur[b0 + n] = code;
                    a.sa.codes_out[(size_t)(b0 + n) * a.sa.Q + pos] = (int64_t)code;
                    if (pos == n_pos - 1) a.sa.frame_ctr[key.slot] = (int32_t)key.frame_no + 1;
                }
                if (i + 1 < mine) dt_bar();   // the sampler's scratch is free again
            }
            fb_stamp(dbg, 13);
        }
        w.linger();
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == DT_CONSUMERS / 32 + 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

}  // namespace vuib
