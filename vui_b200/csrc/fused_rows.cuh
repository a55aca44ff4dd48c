// The two-kernel transformer layer of fused_blocks.cuh for two to four rows (streams) at once.
//
// Four streams need the same weights as one, so what bounds them is the same chain of exchanges; five kernels a layer on
// register-tile GEMVs paid 26 us for a backbone layer at three streams, where one stream's two kernels pay 12.  The split over
// clusters and CTAs, the exchanges and the rounding points are those of the single-row kernels; what the rows change:
//   * matrix rows in shared memory are read once for all streams: mma.sync m16n8k16 with the streams as columns, each twice, for
//     the two rotations of the k blocks that keep the reads free of bank conflicts (mma_rows4);
//   * partial rows are [part][row][K], added up once per cluster (RowSlice);
//   * attention gives each row two warps of every CTA (backbone) or one (depth loop).
// A row's result does not depend on how many rows run beside it.
#pragma once
#include "fused_blocks.cuh"

namespace vuib {

constexpr int FR_ROWS = 4;
constexpr int FR_PAD = 32;        // elements between staged rows, so that neighbouring rows lie in different banks
constexpr int FR_MAX_PARTS = 12;
constexpr int FR_ATT_PRE = 64;    // keys of a row that a CTA requests before use (512 in a cluster)
constexpr int FR_ATT_TH = 256;    // threads of the backbone's attention block; 512 halve a warp's keys, but the block took 8.3 us instead of 6.2

__device__ __forceinline__ void push_f32x4(uint32_t dst, uint32_t bar, const float (&v)[4]) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];"
                 ::"r"(dst), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "r"(bar) : "memory");
}

// The residual rows x_in + bf16(sum_p parts[p]), put together by the cluster: a CTA adds up an eighth of the columns of every row
// and sends the bf16 results to all eight CTAs.  Every CTA adding up whole rows, as the single-row kernels do, took 3.5 us for four
// backbone rows (200 KB from the L2 into each SM); the eighth takes what one row takes, and the exchange 0.4 us.
template <int K>
struct RowSlice {
    static constexpr int TPR = K / FB_CL / 2;   // threads of a row's slice, two columns each
    int r, c;
    bool live;
    unsigned x;                                 // two bf16
    __device__ __forceinline__ void load(const bf16* x_in, int x_stride, const float* parts, int n_parts, int rows, int rank) {
        r = threadIdx.x / TPR;
        c = rank * (K / FB_CL) + 2 * (threadIdx.x % TPR);
        live = r < rows;
        if (!live) return;
        x = __ldcg(reinterpret_cast<const unsigned*>(x_in + (size_t)r * x_stride + c));
        float2 p[FR_MAX_PARTS];
#pragma unroll
        for (int u = 0; u < FR_MAX_PARTS; ++u)
            p[u] = u < n_parts ? __ldcg(reinterpret_cast<const float2*>(parts + ((size_t)u * rows + r) * K + c)) : make_float2(0.f, 0.f);
        if (n_parts > 0) {
            float s0 = 0.f, s1 = 0.f;
#pragma unroll
            for (int u = 0; u < FR_MAX_PARTS; ++u) { s0 += p[u].x; s1 += p[u].y; }
            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x));
            const __nv_bfloat162 h = __floats2bfloat162_rn(f.x + rbf(s0), f.y + rbf(s1));
            x = *reinterpret_cast<const unsigned*>(&h);
        }
    }
    // after cluster_wait(): into row r of every CTA's xs
    __device__ __forceinline__ void send(bf16* xs, uint64_t* bar) const {
        if (!live) return;
#pragma unroll
        for (int peer = 0; peer < FB_CL; ++peer)
            asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];"
                         ::"r"(peer_addr(xs + r * (K + FR_PAD) + c, peer)), "r"(x), "r"(peer_addr(bar, peer)) : "memory");
    }
    __device__ __forceinline__ void store(bf16* out) const {
        if (live) *reinterpret_cast<unsigned*>(out + (size_t)r * K + c) = x;
    }
};

// RMSNorm of the rows in shared memory, in place: a row's warps (TH / 128 of them) take whole pieces of eight columns.
template <int K, int TH>
struct RowNorm {
    static constexpr int WPR = TH / 32 / FR_ROWS;
    static constexpr int NCH = K / WPR / 256;
    static_assert(NCH * WPR * 256 == K && WPR >= 1, "sixteen or eight columns a thread");
    uint4 w[NCH];
    __device__ __forceinline__ int col(int i) const {
        return ((threadIdx.x >> 5) % WPR) * (K / WPR) + i * 256 + (threadIdx.x & 31) * 8;
    }
    __device__ __forceinline__ void preload(const bf16* norm_w) {
#pragma unroll
        for (int i = 0; i < NCH; ++i) w[i] = __ldg(reinterpret_cast<const uint4*>(norm_w + col(i)));
    }
    __device__ __forceinline__ void run(bf16* xs, float eps, int rows, float* red) const {
        const int warp = threadIdx.x >> 5, r = warp / WPR;
        bf16* row = xs + r * (K + FR_PAD);
        float v[NCH][8], ss = 0.f;
        if (r < rows) {
#pragma unroll
            for (int i = 0; i < NCH; ++i) {
                unpack8(*reinterpret_cast<const uint4*>(row + col(i)), v[i]);
#pragma unroll
                for (int j = 0; j < 8; ++j) ss = fmaf(v[i][j], v[i][j], ss);
            }
            ss = warp_sum(ss);
            if ((threadIdx.x & 31) == 0) red[warp] = ss;
        }
        __syncthreads();
        if (r < rows) {
            float tot = 0.f;
#pragma unroll
            for (int i = 0; i < WPR; ++i) tot += red[r * WPR + i];
            const float rinv = rsqrtf(tot / (float)K + eps);
#pragma unroll
            for (int i = 0; i < NCH; ++i) {
                float wf[8], o[8];
                unpack8(w[i], wf);
#pragma unroll
                for (int j = 0; j < 8; ++j) o[j] = rbf(v[i][j] * rinv) * wf[j];
                *reinterpret_cast<uint4*>(row + col(i)) = pack8(o);
            }
        }
        __syncthreads();
    }
};

// mma_rows (fused_blocks.cuh) for four streams: matrix row g of a tile visits the k blocks of the warp's slice rotated by g & 1;
// column c carries stream c & 3 at the blocks rotated by c >> 2, so row g's sums are columns (g & 1) * 4 .. + 3.
// Partial sums land in red[warp][row][stream].  Columns of streams that do not exist hold what shared memory held: never read.
template <int K, int NROWS, int NW>
__device__ __forceinline__ void mma_rows4(const bf16* mat, const bf16* xs, float* red, int warp, int lane) {
    constexpr int NT = (NROWS + 15) / 16;
    constexpr int NBS = K / 32 / NW;
    static_assert(K % (32 * NW) == 0 && NBS >= 2 && NBS % 2 == 0, "every warp takes an even number of blocks");
    const int g = lane >> 2, t = lane & 3;
    float d[NT][4];
#pragma unroll
    for (int i = 0; i < NT; ++i) d[i][0] = d[i][1] = d[i][2] = d[i][3] = 0.f;
#pragma unroll
    for (int i = 0; i < NBS; ++i) {
        const int ka = (warp * NBS + ((i + (g & 1)) % NBS)) * 32 + 8 * t;
        const int kx = (warp * NBS + ((i + (g >> 2)) % NBS)) * 32 + 8 * t;
        const uint4 hb = *reinterpret_cast<const uint4*>(xs + (g & 3) * (K + FR_PAD) + kx);
#pragma unroll
        for (int tl = 0; tl < NT; ++tl) {
            const int r0 = min(tl * 16 + g, NROWS - 1), r1 = min(tl * 16 + 8 + g, NROWS - 1);
            const uint4 w0 = *reinterpret_cast<const uint4*>(mat + (size_t)r0 * K + ka);
            const uint4 w1 = *reinterpret_cast<const uint4*>(mat + (size_t)r1 * K + ka);
            asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                         : "+f"(d[tl][0]), "+f"(d[tl][1]), "+f"(d[tl][2]), "+f"(d[tl][3])
                         : "r"(w0.x), "r"(w1.x), "r"(w0.y), "r"(w1.y), "r"(hb.x), "r"(hb.y));
            asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                         : "+f"(d[tl][0]), "+f"(d[tl][1]), "+f"(d[tl][2]), "+f"(d[tl][3])
                         : "r"(w0.z), "r"(w1.z), "r"(w0.w), "r"(w1.w), "r"(hb.z), "r"(hb.w));
        }
    }
    if ((t >> 1) == (g & 1)) {   // columns 2t, 2t + 1 are streams (t & 1) * 2 and the next, at this row's rotation
        float2* to = reinterpret_cast<float2*>(red) + ((size_t)warp * (NT * 16) + g) * 2 + (t & 1);
#pragma unroll
        for (int tl = 0; tl < NT; ++tl) {
            to[(tl * 16) * 2] = make_float2(d[tl][0], d[tl][1]);
            to[(tl * 16 + 8) * 2] = make_float2(d[tl][2], d[tl][3]);
        }
    }
}
template <int NROWS, int NW>
__device__ __forceinline__ float mma_rows4_total(const float* red, int r, int n) {
    constexpr int NT = (NROWS + 15) / 16;
    float s[NW];
#pragma unroll
    for (int w = 0; w < NW; ++w) s[w] = red[(w * (NT * 16) + r) * FR_ROWS + n];
#pragma unroll
    for (int k = NW / 2; k > 0; k /= 2)   // as a tree: a chain of NW additions is 16 x 4 cycles
#pragma unroll
        for (int w = 0; w < k; ++w) s[w] += s[w + k];
    return s[0];
}

// A column slice of out_proj or w2 (ROWS x C in shared memory) times the streams' vectors (bf16, C + FR_PAD apart), a warp for every
// 16 rows; stream n's results go to out + n * out_stride.  As dot products with the vectors in registers this took 1.9 us of the
// backbone's MLP block at four streams, on the tensor cores 0.5 us.
template <int C, int ROWS, int NW>
__device__ __forceinline__ void mma_slice4(const bf16* mat, const bf16* vec, int rows, float* out, size_t out_stride, int warp, int lane) {
    constexpr int NB = C / 32;
    static_assert(C % 64 == 0 && ROWS % 16 == 0 && ROWS / 16 <= NW, "a tile of 16 rows per warp, an even number of k blocks");
    if (warp >= ROWS / 16) return;
    const int g = lane >> 2, t = lane & 3;
    const bf16* m0 = mat + (size_t)(warp * 16 + g) * C + 8 * t;
    const bf16* v0 = vec + (g & 3) * (C + FR_PAD) + 8 * t;
    float d0[4] = {0.f, 0.f, 0.f, 0.f}, d1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        const int ka = ((i + (g & 1)) % NB) * 32, kx = ((i + (g >> 2)) % NB) * 32;
        const uint4 hb = *reinterpret_cast<const uint4*>(v0 + kx);
        const uint4 w0 = *reinterpret_cast<const uint4*>(m0 + ka);
        const uint4 w1 = *reinterpret_cast<const uint4*>(m0 + 8 * C + ka);
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(d0[0]), "+f"(d0[1]), "+f"(d0[2]), "+f"(d0[3])
                     : "r"(w0.x), "r"(w1.x), "r"(w0.y), "r"(w1.y), "r"(hb.x), "r"(hb.y));
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(d1[0]), "+f"(d1[1]), "+f"(d1[2]), "+f"(d1[3])
                     : "r"(w0.z), "r"(w1.z), "r"(w0.w), "r"(w1.w), "r"(hb.z), "r"(hb.w));
    }
    if ((t >> 1) != (g & 1)) return;
    float* o = out + (size_t)((t & 1) * 2) * out_stride + warp * 16 + g;
    if ((t & 1) * 2 < rows) { o[0] = d0[0] + d1[0]; o[8] = d0[2] + d1[2]; }
    if ((t & 1) * 2 + 1 < rows) { o[out_stride] = d0[1] + d1[1]; o[out_stride + 8] = d0[3] + d1[3]; }
}

// ---------------------------------------------------------------------------
// Attention block.  AttnBlockArgs with rows: x_in rows are x_stride elements apart, x_out and tap (rows, K),
// parts_in / parts_out [part][rows][K]; the depth loop's row n uses slot n at fixed_pos,
// or with `pairs` (fixed_pos = 0 only) position n & 1 of slot n / 2.
// ---------------------------------------------------------------------------
template <int K, int G, bool SHORT, int TH>
struct AttnRowsSmem {
    static constexpr int QR = G * HD / FB_CL;
    static constexpr int KR = HD / FB_CL;
    static constexpr int NR = QR + 2 * KR;
    static constexpr int NP = NR / 2;
    static constexpr int OR = K / FB_CL;
    static constexpr int OC = G * HD;
    static constexpr int QKV = G * HD + 2 * HD;
    static constexpr int PS = HD + 4;            // a partial state: acc[64], m, l; acc is pushed in pieces of four
    alignas(128) bf16 wo[OR * OC];
    alignas(16) bf16 w[NR * K];
    alignas(16) bf16 xs[FR_ROWS * (K + FR_PAD)];
    alignas(16) float qkv[FR_ROWS * QKV];
    alignas(16) float part[SHORT ? 4 : FB_CL * FR_ROWS * G * PS];
    float wpart[SHORT ? 1 : TH / 32][G][8][10];
    alignas(16) bf16 attn[FR_ROWS * (OC + FR_PAD)];
    float s_new[FR_ROWS][G];
    float red[TH / 32];
    alignas(16) float dots[(TH / 32) * ((NR + 15) / 16) * 16 * FR_ROWS];
    alignas(8) uint64_t bar;
    alignas(8) uint64_t bar_x;     // residual rows complete
    alignas(8) uint64_t bar_qkv;
    alignas(8) uint64_t bar_part;
};

template <int K, int G, bool SHORT, int TH>
__global__ void __launch_bounds__(TH, 1) k_attn_rows(const __grid_constant__ CUtensorMap map_wo, AttnBlockArgs a) {
    using S = AttnRowsSmem<K, G, SHORT, TH>;
    constexpr int NW = TH / 32, WPR = SHORT ? 1 : NW / FR_ROWS;   // warps of the CTA, warps for a row's keys
    static_assert(!SHORT || G == 1, "the short form handles one query head per cluster");
    static_assert(SHORT || (G == 2 && WPR >= 2 && TH % 128 == 0), "two of a row's warps score the new key for a head each");
    constexpr int QR = S::QR, KR = S::KR, OR = S::OR, OC = S::OC, NP = S::NP, QKV = S::QKV, PS = S::PS;
    constexpr int NPRE = SHORT ? 4 : FR_ATT_PRE / WPR / 4;
    static_assert(NP * 16 <= TH, "sixteen threads finish each row pair, four a stream");
    extern __shared__ __align__(128) unsigned char fb_smem[];
    S& sm = *reinterpret_cast<S*>(fb_smem);
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int kvh = blockIdx.x / FB_CL;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int qcols = a.Hq * HD, kvcols = a.Hkv * HD, rows = a.rows;
    fb_stamp(a.dbg, 0);
    pdl_trigger();

    if (tid == 0) {
        mbar_init(&sm.bar, 1);
        mbar_init(&sm.bar_x, 1);
        mbar_init(&sm.bar_qkv, 1);
        mbar_init(&sm.bar_part, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_expect_tx(&sm.bar_x, (uint32_t)(rows * K * 2));
        mbar_expect_tx(&sm.bar_qkv, (uint32_t)(rows * QKV * 4));
        if (!SHORT) mbar_expect_tx(&sm.bar_part, (uint32_t)(FB_CL * rows * G * (HD + 2) * 4));
    }
    __syncthreads();
    cluster_arrive_relaxed();   // before the weight copies (see k_attn_block)
    if (tid == 0) {
        mbar_expect_tx(&sm.bar, (uint32_t)(S::NR * K * 2 + OR * OC * 2));
        bulk_g2s(sm.w, a.wqkv + (size_t)(kvh * G * HD + rank * QR) * K, QR * K * 2, &sm.bar);
        bulk_g2s(sm.w + QR * K, a.wqkv + (size_t)(qcols + kvh * HD + rank * KR) * K, KR * K * 2, &sm.bar);
        bulk_g2s(sm.w + (QR + KR) * K, a.wqkv + (size_t)(qcols + kvcols + kvh * HD + rank * KR) * K, KR * K * 2, &sm.bar);
        tma_load_2d(sm.wo, &map_wo, kvh * OC, rank * OR, &sm.bar);
    }
    RowNorm<K, TH> norm;
    norm.preload(a.norm_w);

    // ---- what this thread finishes later: one stream of one q/k/v row pair, for a quarter of the cluster's CTAs
    const int pn = (tid >> 2) & 3;
    const bool pair_live = (tid >> 4) < NP && pn < rows;
    const int prow = 2 * (pair_live ? tid >> 4 : 0);
    const bool is_q = prow < QR, is_k = !is_q && prow < QR + KR;
    const int sub = is_q ? prow : (is_k ? prow - QR : prow - QR - KR);
    const int pairs = SHORT && a.pairs ? 1 : 0;
    int pslot = pn >> pairs, ppos = a.fixed_pos + (pn & pairs);
    float c0 = 1.f, s0 = 0.f, c1 = 1.f, s1 = 0.f;
    // ---- and its keys: a quarter of every CTA's warps for a row (backbone), one (depth loop)
    const int s8 = lane & 7, g4 = lane >> 3;
    const int arow = warp / WPR, asub = warp % WPR;
    const bool row_live = arow < rows;
    const size_t pos_stride = (size_t)kvcols;
    int slot = arow >> pairs, pos = a.fixed_pos;   // old keys: those before the pair
    int t_begin = 0, t_end = 0;
    const bf16* kb = nullptr;
    const bf16* vb = nullptr;
    uint4 kr[NPRE], vr[NPRE];
    auto key_of = [&](int it) { return SHORT ? it * 4 + g4 : t_begin + (it * WPR + asub) * 4 + g4; };
    auto request = [&](int sl, int ps) {
        slot = sl;
        pos = ps;
        const int n_old = SHORT ? min(pos, 16) : pos;
        const int chunk = SHORT ? n_old : (n_old + FB_CL - 1) / FB_CL;
        t_begin = SHORT ? 0 : rank * chunk;
        t_end = row_live ? min(n_old, t_begin + chunk) : 0;
        const size_t base = (size_t)(row_live ? slot : 0) * a.max_seq * pos_stride + kvh * HD + s8 * 8;
        kb = a.k_cache + base;
        vb = a.v_cache + base;
#pragma unroll
        for (int it = 0; it < NPRE; ++it) {
            const int t = key_of(it);
            const bool ok = t < t_end;
            kr[it] = ok ? ld_l2(kb + (size_t)t * pos_stride) : make_uint4(0, 0, 0, 0);
            vr[it] = ok ? ld_l2(vb + (size_t)t * pos_stride) : make_uint4(0, 0, 0, 0);
        }
    };
    bool early = false;
    if constexpr (!SHORT) {   // before the dependency wait, with the position as memory has it now (see k_attn_block)
        const int r = row_live ? arow : 0;
        int sg = __ldcg(a.row_slot + r), pg = __ldcg(a.row_pos + r);
        sg = sg < 0 ? 0 : (sg >= a.n_slots ? a.n_slots - 1 : sg);
        pg = pg < 0 ? 0 : (pg >= a.max_seq ? a.max_seq - 1 : pg);
        request(sg, pg);
        early = true;
    }
    pdl_wait();
    fb_stamp(a.dbg, 1);

    int sl = arow >> pairs, ps = a.fixed_pos;
    if constexpr (!SHORT) {
        const int r = row_live ? arow : 0;
        sl = __ldcg(a.row_slot + r);
        ps = __ldcg(a.row_pos + r);
        pslot = __ldcg(a.row_slot + (pair_live ? pn : 0));
        ppos = __ldcg(a.row_pos + (pair_live ? pn : 0));
    }
    RowSlice<K> slice;
    slice.load(a.x_in, a.x_stride, a.parts_in, a.n_parts_in, rows, rank);
    if (!early || sl != slot || ps != pos) request(sl, ps);
    if (a.rope && (is_q || is_k)) {
        const int dd = (is_q ? rank * QR + sub : rank * KR + sub) & (HD - 1);
        const uint2 f = __ldg(reinterpret_cast<const uint2*>(a.rope + ((size_t)ppos * HD + dd) * 2));
        c0 = bf2f(__ushort_as_bfloat16((unsigned short)(f.x & 0xffffu)));
        s0 = bf2f(__ushort_as_bfloat16((unsigned short)(f.x >> 16)));
        c1 = bf2f(__ushort_as_bfloat16((unsigned short)(f.y & 0xffffu)));
        s1 = bf2f(__ushort_as_bfloat16((unsigned short)(f.y >> 16)));
    }
    fb_stamp(a.dbg, 8);
    cluster_wait();
    slice.send(sm.xs, &sm.bar_x);
    if (kvh == 0) {
        slice.store(a.x_out);
        if (a.tap) slice.store(a.tap);
    }
    if (!wait_pushed(&sm.bar_x, a.spin_limit) && tid == 0) atomicOr(a.flag, FLAG_COPY_TIMEOUT);
    norm.run(sm.xs, a.eps, rows, sm.red);
    fb_stamp(a.dbg, 2);
    wait_weights(&sm.bar, a.spin_limit, a.flag);
    fb_stamp(a.dbg, 3);

    // ---- q/k/v rows of this CTA for every stream, results to every CTA of the cluster
    mma_rows4<K, S::NR, NW>(sm.w, sm.xs, sm.dots, warp, lane);
    __syncthreads();
    if (pair_live) {
        float t0 = rbf(mma_rows4_total<S::NR, NW>(sm.dots, prow, pn));
        float t1 = rbf(mma_rows4_total<S::NR, NW>(sm.dots, prow + 1, pn));
        if (a.rope && (is_q || is_k)) {
            const float o0 = rbf(rbf(t0 * c0) + rbf((-t1) * s0));
            const float o1 = rbf(rbf(t1 * c1) + rbf(t0 * s1));
            t0 = o0;
            t1 = o1;
        }
        const int idx = pn * QKV + (is_q ? rank * QR + sub : (is_k ? G * HD : G * HD + HD) + rank * KR + sub);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int peer = (tid & 3) * 2 + i;
            push_f32x2(peer_addr(sm.qkv + idx, peer), peer_addr(&sm.bar_qkv, peer), t0, t1);
        }
        if (!is_q && (tid & 3) == 0) {
            bf16* cache = is_k ? a.k_cache : a.v_cache;
            *reinterpret_cast<__nv_bfloat162*>(cache + ((size_t)pslot * a.max_seq + ppos) * pos_stride + kvh * HD + rank * KR + sub) =
                __floats2bfloat162_rn(t0, t1);
        }
    }
    fb_stamp(a.dbg, 9);
    if (!wait_pushed(&sm.bar_qkv, a.spin_limit) && tid == 0) atomicOr(a.flag, FLAG_COPY_TIMEOUT);
    fb_stamp(a.dbg, 4);

    // ---- attention: scores of the requested keys first, one maximum, then the weighted sum
    const float* qkv = sm.qkv + (row_live ? arow : 0) * QKV;
    float qf[G][8];
#pragma unroll
    for (int h = 0; h < G; ++h) {
        const float4 q0 = *reinterpret_cast<const float4*>(qkv + h * HD + s8 * 8);
        const float4 q1 = *reinterpret_cast<const float4*>(qkv + h * HD + s8 * 8 + 4);
        qf[h][0] = q0.x; qf[h][1] = q0.y; qf[h][2] = q0.z; qf[h][3] = q0.w;
        qf[h][4] = q1.x; qf[h][5] = q1.y; qf[h][6] = q1.z; qf[h][7] = q1.w;
    }
    if constexpr (SHORT) {
        if (row_live && (arow & pairs)) {   // the second of a pair (of which no key is in the cache) also sees the first one's key
            const float* first = qkv - QKV + HD + s8 * 8;
            float kf[8], vf[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) { kf[j] = first[j]; vf[j] = first[HD + j]; }
            kr[0] = pack8(kf);
            vr[0] = pack8(vf);
            t_end = 1;
        }
    }
    float m[G], l[G], acc[G][8], sc[G][NPRE];
#pragma unroll
    for (int it = 0; it < NPRE; ++it) {
        float kf[8];
        unpack8(kr[it], kf);
#pragma unroll
        for (int h = 0; h < G; ++h) {
            float d = 0.f;
#pragma unroll
            for (int j = 0; j < 8; ++j) d = fmaf(qf[h][j], kf[j], d);
            sc[h][it] = d;
        }
    }
    float dn = 0.f;   // depth loop: the new key, counted once, by the first key group
    if constexpr (SHORT) {
#pragma unroll
        for (int j = 0; j < 8; ++j) dn = fmaf(qf[0][j], qkv[HD + s8 * 8 + j], dn);
    }
#pragma unroll
    for (int o = 1; o <= 4; o <<= 1) {
#pragma unroll
        for (int h = 0; h < G; ++h)
#pragma unroll
            for (int it = 0; it < NPRE; ++it) sc[h][it] += __shfl_xor_sync(0xffffffffu, sc[h][it], o);
        if constexpr (SHORT) dn += __shfl_xor_sync(0xffffffffu, dn, o);
    }
#pragma unroll
    for (int h = 0; h < G; ++h) {
        const float sn = SHORT && g4 == 0 ? dn * 0.125f : NEG_BIG;
        m[h] = sn;
#pragma unroll
        for (int it = 0; it < NPRE; ++it) {
            sc[h][it] = key_of(it) < t_end ? sc[h][it] * 0.125f : NEG_BIG;
            m[h] = fmaxf(m[h], sc[h][it]);
        }
        m[h] = fmaxf(m[h], __shfl_xor_sync(0xffffffffu, m[h], 8));
        m[h] = fmaxf(m[h], __shfl_xor_sync(0xffffffffu, m[h], 16));
        const float pnew = SHORT && g4 == 0 ? __expf(sn - m[h]) : 0.f;
        l[h] = pnew;
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[h][j] = SHORT ? pnew * qkv[2 * HD + s8 * 8 + j] : 0.f;
#pragma unroll
        for (int it = 0; it < NPRE; ++it) {
            sc[h][it] = key_of(it) < t_end ? __expf(sc[h][it] - m[h]) : 0.f;
            l[h] += sc[h][it];
        }
    }
#pragma unroll
    for (int it = 0; it < NPRE; ++it) {
        float vf[8];
        unpack8(vr[it], vf);
#pragma unroll
        for (int h = 0; h < G; ++h)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[h][j] = fmaf(sc[h][it], vf[j], acc[h][j]);
    }
    if constexpr (SHORT) {
#pragma unroll
        for (int o = 8; o <= 16; o <<= 1) {
            l[0] += __shfl_xor_sync(0xffffffffu, l[0], o);
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[0][j] += __shfl_xor_sync(0xffffffffu, acc[0][j], o);
        }
        if (row_live && g4 == 0) {
            const float inv = 1.f / l[0];
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[0][j] *= inv;
            *reinterpret_cast<uint4*>(sm.attn + arow * (OC + FR_PAD) + s8 * 8) = pack8(acc[0]);
        }
    } else {
        if (row_live && asub < G) {   // score of the new key (this step's own position): two of the row's warps, a q head each
            const float* q = qkv + asub * HD;
            const float* kn = qkv + G * HD;
            float d = q[lane] * kn[lane] + q[lane + 32] * kn[lane + 32];
            d = warp_sum(d);
            if (lane == 0) sm.s_new[arow][asub] = d * 0.125f;
        }
        for (int tb = t_begin + NPRE * WPR * 4; tb < t_end; tb += WPR * 4) {   // longer caches: the rest, block by block (uniform over the warp)
            const int t = tb + asub * 4 + g4;
            const bool ok = t < t_end;
            float kf[8], vf[8];
            unpack8(ok ? ld_l2(kb + (size_t)t * pos_stride) : make_uint4(0, 0, 0, 0), kf);
            unpack8(ok ? ld_l2(vb + (size_t)t * pos_stride) : make_uint4(0, 0, 0, 0), vf);
#pragma unroll
            for (int h = 0; h < G; ++h) {
                float d = 0.f;
#pragma unroll
                for (int j = 0; j < 8; ++j) d = fmaf(qf[h][j], kf[j], d);
                d += __shfl_xor_sync(0xffffffffu, d, 1);
                d += __shfl_xor_sync(0xffffffffu, d, 2);
                d += __shfl_xor_sync(0xffffffffu, d, 4);
                if (ok) {
                    const float s = d * 0.125f, mn = fmaxf(m[h], s);
                    const float corr = __expf(m[h] - mn), p = __expf(s - mn);
                    l[h] = l[h] * corr + p;
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[h][j] = fmaf(p, vf[j], acc[h][j] * corr);
                    m[h] = mn;
                }
            }
        }
        // merge the warp's four key groups, then the row's warps, then the cluster's CTAs
        if (t_begin + NPRE * WPR * 4 < t_end) {   // only those further keys leave the groups with different maxima
#pragma unroll
            for (int h = 0; h < G; ++h) {
                float mx = fmaxf(m[h], __shfl_xor_sync(0xffffffffu, m[h], 8));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                const float c = __expf(m[h] - mx);
                m[h] = mx;
                l[h] *= c;
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[h][j] *= c;
            }
        }
#pragma unroll
        for (int o = 8; o <= 16; o <<= 1) {
#pragma unroll
            for (int h = 0; h < G; ++h) {
                l[h] += __shfl_xor_sync(0xffffffffu, l[h], o);
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[h][j] += __shfl_xor_sync(0xffffffffu, acc[h][j], o);
            }
        }
        if (g4 == 0) {
#pragma unroll
            for (int h = 0; h < G; ++h) {
#pragma unroll
                for (int j = 0; j < 8; ++j) sm.wpart[warp][h][s8][j] = acc[h][j];
                sm.wpart[warp][h][s8][8] = m[h];
                sm.wpart[warp][h][s8][9] = l[h];
            }
        }
        __syncthreads();
        fb_stamp(a.dbg, 10);
        {   // thread: four dims of one (row, head), to some of the cluster's CTAs
            const int u = tid & 127, r = u >> 5, h = (u >> 4) & 1, d4 = (u & 15) * 4;
            if (r < rows) {
                const float* w[WPR];
                const int dj = d4 & 7;
                float M_ = NEG_BIG, L_ = 0.f, v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int i = 0; i < WPR; ++i) {
                    w[i] = sm.wpart[r * WPR + i][h][d4 >> 3];
                    M_ = fmaxf(M_, w[i][8]);
                }
#pragma unroll
                for (int i = 0; i < WPR; ++i) {
                    const float e = __expf(w[i][8] - M_);
                    L_ += w[i][9] * e;
#pragma unroll
                    for (int j = 0; j < 4; ++j) v[j] += w[i][dj + j] * e;
                }
                float* mine = sm.part + ((rank * FR_ROWS + r) * G + h) * PS;
#pragma unroll
                for (int i = 0; i < FB_CL * 128 / TH; ++i) {
                    const int c = (tid >> 7) * (FB_CL * 128 / TH) + i;
                    const uint32_t pbar = peer_addr(&sm.bar_part, c);
                    push_f32x4(peer_addr(mine + d4, c), pbar, v);
                    if (d4 == 0) push_f32x2(peer_addr(mine + HD, c), pbar, M_, L_);
                }
            }
        }
        fb_stamp(a.dbg, 11);
        if (!wait_pushed(&sm.bar_part, a.spin_limit) && tid == 0) atomicOr(a.flag, FLAG_COPY_TIMEOUT);
        fb_stamp(a.dbg, 5);
        for (int o = tid; o < rows * G * HD; o += TH) {   // every CTA merges in CTA order, then the new key: same bits everywhere
            const int r = o / (G * HD), h = (o / HD) % G, dim = o % HD;
            const float* p = sm.part + (r * G + h) * PS;
            const float sn = sm.s_new[r][h];
            float Mx = sn;
#pragma unroll
            for (int c = 0; c < FB_CL; ++c) Mx = fmaxf(Mx, p[c * FR_ROWS * G * PS + HD]);
            float Ls = 0.f, Os = 0.f;
#pragma unroll
            for (int c = 0; c < FB_CL; ++c) {
                const float e = __expf(p[c * FR_ROWS * G * PS + HD] - Mx);
                Ls += p[c * FR_ROWS * G * PS + HD + 1] * e;
                Os += p[c * FR_ROWS * G * PS + dim] * e;
            }
            const float en = __expf(sn - Mx);
            Ls += en;
            Os += en * sm.qkv[r * QKV + G * HD + HD + dim];
            sm.attn[r * (OC + FR_PAD) + h * HD + dim] = __float2bfloat16_rn(Os / Ls);
        }
    }
    __syncthreads();
    fb_stamp(a.dbg, 12);

    // ---- this head group's K-slice of out_proj for the CTA's rows
    mma_slice4<OC, OR, NW>(sm.wo, sm.attn, rows, a.parts_out + (size_t)kvh * rows * K + rank * OR, (size_t)K, warp, lane);
    fb_stamp(a.dbg, 6);
}

// ---------------------------------------------------------------------------
// MLP block
// ---------------------------------------------------------------------------
template <int K, int F, int U, int TH>
struct MlpRowsSmem {
    static constexpr int CU = U * FB_CL;
    static constexpr int OR = K / FB_CL;
    static constexpr int NCL = F / CU;
    static_assert(F % CU == 0 && CU % 8 == 0 && NCL <= FR_MAX_PARTS, "ffn must split evenly into 16-byte pieces, over at most 12 clusters");
    alignas(128) bf16 w2[OR * CU];
    alignas(16) bf16 w13[2 * U * K];
    alignas(16) bf16 xs[FR_ROWS * (K + FR_PAD)];
    alignas(16) bf16 g[FR_ROWS * (CU + FR_PAD)];
    float red[TH / 32];
    alignas(16) float dots[(TH / 32) * ((2 * U + 15) / 16) * 16 * FR_ROWS];
    alignas(8) uint64_t bar;
    alignas(8) uint64_t bar_x;
    alignas(8) uint64_t bar_g;
    alignas(8) uint64_t bar_w2;
};

template <int K, int F, int U, int TH>
__global__ void __launch_bounds__(TH, 1) k_mlp_rows(const __grid_constant__ CUtensorMap map_w2, MlpBlockArgs a) {
    using S = MlpRowsSmem<K, F, U, TH>;
    constexpr int NWARP = TH / 32;
    constexpr int CU = S::CU, OR = S::OR;
    constexpr bool LATE_W2 = K >= 1024;   // see k_mlp_block
    static_assert(U * 16 == TH, "sixteen threads finish each hidden unit, four a stream");
    extern __shared__ __align__(128) unsigned char fb_smem[];
    S& sm = *reinterpret_cast<S*>(fb_smem);
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int cid = blockIdx.x / FB_CL;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, rows = a.rows;
    fb_stamp(a.dbg, 0);
    pdl_trigger();

    if (tid == 0) {
        mbar_init(&sm.bar, 1);
        mbar_init(&sm.bar_x, 1);
        mbar_init(&sm.bar_g, 1);
        mbar_init(&sm.bar_w2, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_expect_tx(&sm.bar_x, (uint32_t)(rows * K * 2));
        mbar_expect_tx(&sm.bar_g, (uint32_t)(rows * CU * 2));
    }
    __syncthreads();
    cluster_arrive_relaxed();
    if (tid == 0) {
        mbar_expect_tx(&sm.bar, (uint32_t)(2 * U * K * 2 + (LATE_W2 ? 0 : OR * CU * 2)));
        const size_t u0 = (size_t)cid * CU + rank * U;
        bulk_g2s(sm.w13, a.w1 + u0 * K, U * K * 2, &sm.bar);
        bulk_g2s(sm.w13 + U * K, a.w3 + u0 * K, U * K * 2, &sm.bar);
        if constexpr (!LATE_W2) tma_load_2d(sm.w2, &map_w2, cid * CU, rank * OR, &sm.bar);
    }
    if (cid < FB_HINT_CLUSTERS) prefetch_l2(a.next, TH);
    RowNorm<K, TH> norm;
    norm.preload(a.norm_w);
    if (a.next_k && cid < FB_HINT_CLUSTERS) {   // the next layer's K/V rows into the L2 (see k_mlp_block)
        const size_t row_bytes = (size_t)a.kvcols * sizeof(bf16);
        const size_t n_hint = (size_t)(gridDim.x < FB_HINT_CLUSTERS * FB_CL ? gridDim.x : FB_HINT_CLUSTERS * FB_CL) * TH;
        for (int r = 0; r < rows; ++r) {
            int slot = __ldcg(a.row_slot + r), pos = __ldcg(a.row_pos + r);
            slot = slot < 0 ? 0 : (slot >= a.n_slots ? a.n_slots - 1 : slot);
            pos = pos < 0 ? 0 : (pos > a.max_seq ? a.max_seq : pos);
            const size_t lines = (size_t)pos * row_bytes / 128;
            const char* kbase = reinterpret_cast<const char*>(a.next_k) + (size_t)slot * a.max_seq * row_bytes;
            const char* vbase = reinterpret_cast<const char*>(a.next_v) + (size_t)slot * a.max_seq * row_bytes;
            for (size_t i = (size_t)blockIdx.x * TH + tid; i < 2 * lines; i += n_hint) {
                const char* p = i < lines ? kbase + i * 128 : vbase + (i - lines) * 128;
                asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
            }
        }
    }
    pdl_wait();
    fb_stamp(a.dbg, 1);

    RowSlice<K> slice;
    slice.load(a.x_in, K, a.parts_in, a.n_parts_in, rows, rank);
    fb_stamp(a.dbg, 8);
    cluster_wait();
    slice.send(sm.xs, &sm.bar_x);
    if (cid == 0) slice.store(a.x_out);
    if (!wait_pushed(&sm.bar_x, a.spin_limit) && tid == 0) atomicOr(a.flag, FLAG_COPY_TIMEOUT);
    norm.run(sm.xs, a.eps, rows, sm.red);
    fb_stamp(a.dbg, 2);
    if (LATE_W2 && tid == 0) {
        mbar_expect_tx(&sm.bar_w2, (uint32_t)(OR * CU * 2));
        tma_load_2d(sm.w2, &map_w2, cid * CU, rank * OR, &sm.bar_w2);
    }
    wait_weights(&sm.bar, a.spin_limit, a.flag);
    fb_stamp(a.dbg, 3);

    // ---- SiLU(w1 h) * (w3 h) of this CTA's hidden units for every stream; a thread sends a pair of units to one of the cluster's CTAs
    mma_rows4<K, 2 * U, NWARP>(sm.w13, sm.xs, sm.dots, warp, lane);
    __syncthreads();
    {
        const int u = tid >> 4, n = (tid >> 2) & 3;
        float send = 0.f;
        if (n < rows) {
            const float a1 = rbf(mma_rows4_total<2 * U, NWARP>(sm.dots, u, n));
            const float a3 = rbf(mma_rows4_total<2 * U, NWARP>(sm.dots, U + u, n));
            send = rbf(rbf(a1 / (1.0f + expf(-a1))) * a3);
        }
        const float other = __shfl_xor_sync(0xffffffffu, send, 16);   // the unit beside this one: a warp holds two
        if (n < rows) {
            const bool odd = (u & 1) != 0;
            const __nv_bfloat162 h = __floats2bfloat162_rn(odd ? other : send, odd ? send : other);
            const int peer = (tid & 3) * 2 + (odd ? 1 : 0);
            asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];"
                         ::"r"(peer_addr(sm.g + n * (CU + FR_PAD) + rank * U + (u & ~1), peer)),
                           "r"(*reinterpret_cast<const unsigned*>(&h)), "r"(peer_addr(&sm.bar_g, peer)) : "memory");
        }
    }
    fb_stamp(a.dbg, 9);
    if (!wait_pushed(&sm.bar_g, a.spin_limit) && tid == 0) atomicOr(a.flag, FLAG_COPY_TIMEOUT);
    fb_stamp(a.dbg, 4);

    if constexpr (LATE_W2) wait_weights(&sm.bar_w2, a.spin_limit, a.flag);
    mma_slice4<CU, OR, NWARP>(sm.w2, sm.g, rows, a.parts_out + (size_t)cid * rows * K + rank * OR, (size_t)K, warp, lane);
    fb_stamp(a.dbg, 6);
}

}  // namespace vuib
