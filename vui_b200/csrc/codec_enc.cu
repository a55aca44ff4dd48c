// Host side of the codec encoder: workspace layout, weight binding and the launch sequence of one encode call
// (kernels in codec_enc_kernels.cuh).  Entry points: include/vuib200.h, section "Codec encoder".
#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdio.h>
#include <string.h>

#include <new>

#include "../../include/vuib200.h"
#include "codec_enc_kernels.cuh"

using namespace vuie;

struct VuibCodecEnc {
    VuibCodecEncConfig cfg;
    VuibCodecEncWeights w;    // as bound
    VuibCodecEncWeights u;    // with the vectors that are read 16 bytes at a time as the workspace holds them
    unsigned char* ws;
    bool have_ws, have_w, packed;
    int64_t launches;
    size_t off_flag, off_y, off_p[3], off_x, off_q, off_xp, off_gp, off_d, off_dp, off_h, off_rope, off_v, off_w, total;
    struct Packed { vuis::SgWeight c3[4], c1[4], down[4], out, wqkv[VUIB_CODEC_LAYERS], wo[VUIB_CODEC_LAYERS], fc1[VUIB_CODEC_LAYERS],
                    fc2[VUIB_CODEC_LAYERS], half, books; } pk;
    int last_frames, num_sms;
    char err[256];
};

namespace {

int32_t fail(VuibCodecEnc* c, int32_t code, const char* fmt, ...) {
    if (c) {
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(c->err, sizeof(c->err), fmt, ap);
        va_end(ap);
    }
    return code;
}

#define CK(call)                                                                              \
    do {                                                                                      \
        cudaError_t _err = (call);                                                            \
        if (_err != cudaSuccess)                                                              \
            return fail(c, VUIB_ERR_CUDA, "%s failed: %s", #call, cudaGetErrorString(_err));  \
    } while (0)

constexpr int PAD = 8;   // history of a k = 3 or 2-tap convolution, rounded up to the swizzle's period

// Packs the matrices for the split GEMMs (once per binding, on the legacy default stream; binding happens outside any capture).
// Column tiles: 128 where a launch has at least a tile per SM in a 10 s buffer, narrower ones where 250 to 2000 rows leave few.
// They are fixed when the weights are packed, so shorter inputs run with them too: 2 / 16 / 50 / 125 frames take 0.77 / 0.77 / 0.94 /
// 1.47 ms, with tiles half as wide 0.72 / 0.74 / 0.95 / 1.50.
int32_t pack_weights(VuibCodecEnc* c) {
    c->packed = false;
    if (!c->have_ws || !c->have_w) return VUIB_OK;
    const VuibCodecEncConfig& g = c->cfg;
    const VuibCodecEncWeights& w = c->w;
    unsigned char* cur = c->ws + c->off_w;
    cudaError_t e = cudaSuccess;
    auto put = [&](const float* src, int mode, int q0, int q1, int N, int C, int taps, int NT) {
        vuis::SgPack p = {src, nullptr, reinterpret_cast<vuis::bf16*>(cur), mode, q0, q1, N, C, taps, NT};
        if (e == cudaSuccess) e = vuis::sg_pack(p, 0);
        vuis::SgWeight r = {p.out, N, C, taps, NT};
        cur += vuis::sg_weight_bytes(N, C, taps);
        return r;
    };
    int C = g.base_dim;
    const int nt3[4] = {32, 64, 64, 32}, nt1[4] = {64, 128, 128, 64}, ntd[4] = {128, 128, 64, 32};
    for (int i = 0; i < 4; ++i, C *= 2) {
        c->pk.c3[i] = put(w.res[i].c3.w, vuis::SW_ROWS, 0, 0, C / 2, C, 3, nt3[i]);
        c->pk.c1[i] = put(w.res[i].c1.w, vuis::SW_ROWS, 0, 0, C, C / 2, 1, nt1[i]);
        c->pk.down[i] = put(w.down[i].w, vuis::SW_STRIDED, g.ratios[i], C, 2 * C, g.ratios[i] * C, 2, ntd[i]);
    }
    const int D = g.d_model;
    c->pk.out = put(w.conv_out.w, vuis::SW_ROWS, 0, 0, D, C, 3, 32);
    for (int l = 0; l < g.n_layers; ++l) {
        c->pk.wqkv[l] = put(w.layer[l].wqkv, vuis::SW_ROWS, 0, 0, 3 * D, D, 1, 32);
        c->pk.wo[l] = put(w.layer[l].wo, vuis::SW_ROWS, 0, 0, D, D, 1, 32);
        c->pk.fc1[l] = put(w.layer[l].fc1, vuis::SW_ROWS, 0, 0, g.mlp_dim, D, 1, 32);
        c->pk.fc2[l] = put(w.layer[l].fc2, vuis::SW_ROWS, 0, 0, D, g.mlp_dim, 1, 32);
    }
    c->pk.half = put(w.downsample, vuis::SW_STRIDED, 2, D, D, 2 * D, 2, 32);
    c->pk.books = put(w.sem_in, vuis::SW_ROWS, 0, 0, 256, D, 1, 32);   // the acoustic projection's columns follow the semantic one's
    put(w.acq_in, vuis::SW_ROWS, 0, 0, 256, D, 1, 32);
    c->pk.books.N = 512;
    // Biases and layer scales are read 16 bytes at a time and a caller's need not lie that way: they are copied behind one another
    // (their lengths are multiples of 32).
    c->u = w;
    float* vec = reinterpret_cast<float*>(c->ws + c->off_v);
    auto copy = [&](const float*& p, int n) {
        if (e == cudaSuccess) e = cudaMemcpyAsync(vec, p, (size_t)n * 4, cudaMemcpyDeviceToDevice, 0);
        p = vec;
        vec += n;
    };
    C = g.base_dim;
    for (int i = 0; i < 4; ++i, C *= 2) {
        copy(c->u.res[i].c3.b, C / 2);
        copy(c->u.res[i].c1.b, C);
        copy(c->u.down[i].b, 2 * C);
    }
    copy(c->u.conv_out.b, D);
    for (int l = 0; l < g.n_layers; ++l) {
        copy(c->u.layer[l].attn_scale, D);
        copy(c->u.layer[l].mlp_scale, D);
    }
    if (e == cudaSuccess) e = cudaMemsetAsync(c->ws + c->off_flag, 0, 256, 0);
    CK(e);
    const int T25 = g.max_samples / 960;
    vuis::k_srope<<<(T25 * 32 + 255) / 256, 256>>>(w.rope_cos, w.rope_sin, reinterpret_cast<float*>(c->ws + c->off_rope), T25);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(0));
    c->packed = true;
    return VUIB_OK;
}

}  // namespace

extern "C" int32_t vuib_codec_enc_create(const VuibCodecEncConfig* cfg, VuibCodecEnc** out) {
    if (!cfg || !out) return VUIB_ERR_NULL;
    *out = nullptr;
    const VuibCodecEncConfig& g = *cfg;
    bool ok = g.base_dim == 64 && g.ratios[0] == 4 && g.ratios[1] == 5 && g.ratios[2] == 6 && g.ratios[3] == 8 &&
              g.d_model == 512 && g.n_heads == 8 && g.mlp_dim == 2048 && g.n_layers >= 1 &&
              g.n_layers <= VUIB_CODEC_LAYERS;
    if (!ok) return VUIB_ERR_SHAPE;
    if (g.max_samples < 1920 || g.max_samples % 1920 || g.max_samples > 480000) return VUIB_ERR_RANGE;
    VuibCodecEnc* c = new (std::nothrow) VuibCodecEnc();
    if (!c) return VUIB_ERR_NULL;
    memset(c, 0, sizeof(*c));
    c->cfg = g;
    size_t cur = 0;
    auto take = [&](size_t bytes) { size_t o = cur; cur += (bytes + 1023) & ~size_t(1023); return o; };
    const int T0 = g.max_samples, T25 = T0 / 960, T12 = T0 / 1920, D = g.d_model;
    c->off_flag = take(256);
    size_t y = 0, p[3] = {0, 0, 0}, w = 0, v = 0;
    auto most = [](size_t& v, size_t n) { if (n > v) v = n; };
    int C = g.base_dim, T = T0;
    for (int i = 0; i < 4; ++i) {   // a stage: input and its ELU, the residual block's inner half, the strided convolution's input
        most(y, (size_t)C * T * 4);
        most(p[0], vuis::sg_plane_bytes(C, T, PAD));
        most(p[1], vuis::sg_plane_bytes(C / 2, T, PAD));
        most(p[2], vuis::sg_plane_bytes(C * g.ratios[i], T / g.ratios[i], PAD));
        w += vuis::sg_weight_bytes(C / 2, C, 3) + vuis::sg_weight_bytes(C, C / 2, 1) + vuis::sg_weight_bytes(2 * C, 2 * C * g.ratios[i], 1);
        v += C / 2 + C + 2 * C;
        T /= g.ratios[i];
        C *= 2;
    }
    v += D + (size_t)g.n_layers * 2 * D;
    most(p[0], vuis::sg_plane_bytes(C, T, PAD));
    w += vuis::sg_weight_bytes(D, C, 3) + (size_t)g.n_layers * vuis::sg_weight_bytes(4 * D + 2 * g.mlp_dim, D, 1) +
         vuis::sg_weight_bytes(D, 2 * D, 2) + vuis::sg_weight_bytes(512, D, 1);
    c->off_y = take(y);
    for (int i = 0; i < 3; ++i) c->off_p[i] = take(p[i]);
    c->off_x = take((size_t)D * T25 * 4);
    c->off_q = take((size_t)3 * D * T25 * 4);
    c->off_xp = take(vuis::sg_plane_bytes(2 * D, T25, PAD));
    c->off_gp = take(vuis::sg_plane_bytes(g.mlp_dim, T25, PAD));
    c->off_d = take((size_t)D * T12 * 4);
    c->off_dp = take(vuis::sg_plane_bytes(D, T12, PAD));
    c->off_h = take((size_t)512 * T12 * 4);
    c->off_rope = take((size_t)64 * T25 * 4);
    c->off_v = take(v * 4);
    c->off_w = take(w);
    c->total = cur;
    *out = c;
    return VUIB_OK;
}

extern "C" int32_t vuib_codec_enc_destroy(VuibCodecEnc* c) {
    delete c;
    return VUIB_OK;
}

extern "C" int32_t vuib_codec_enc_last_error(VuibCodecEnc* c, char* buf, size_t n) {
    if (!c || !buf || n == 0) return VUIB_ERR_NULL;
    strncpy(buf, c->err, n - 1);
    buf[n - 1] = 0;
    return VUIB_OK;
}

extern "C" int64_t vuib_codec_enc_launch_count(VuibCodecEnc* c) { return c ? c->launches : 0; }

extern "C" int32_t vuib_codec_enc_workspace_bytes(VuibCodecEnc* c, size_t* bytes) {
    if (!c || !bytes) return VUIB_ERR_NULL;
    *bytes = c->total;
    return VUIB_OK;
}

extern "C" int32_t vuib_codec_enc_bind_workspace(VuibCodecEnc* c, void* dev, size_t bytes) {
    if (!c || !dev) return VUIB_ERR_NULL;
    if (bytes < c->total || ((uintptr_t)dev & 255))
        return fail(c, VUIB_ERR_WORKSPACE, "encoder workspace needs %zu bytes, 256-byte aligned; got %zu at %p", c->total,
                    bytes, dev);
    c->ws = static_cast<unsigned char*>(dev);
    c->have_ws = true;
    return pack_weights(c);
}

extern "C" int32_t vuib_codec_enc_bind_weights(VuibCodecEnc* c, const VuibCodecEncWeights* w) {
    if (!c || !w) return VUIB_ERR_NULL;
    VuibCodecEncWeights tmp = *w;
    for (int l = c->cfg.n_layers; l < VUIB_CODEC_LAYERS; ++l) tmp.layer[l] = tmp.layer[0];
    const void* const* p = reinterpret_cast<const void* const*>(&tmp);
    for (size_t i = 0; i < sizeof(tmp) / sizeof(void*); ++i)
        if (!p[i]) return fail(c, VUIB_ERR_NULL, "encoder weight pointer #%zu is NULL", i);
    for (int i = 0; i < 16; ++i)
        if ((uintptr_t)w->codebook[i] & 15) return fail(c, VUIB_ERR_WORKSPACE, "codebook %d is not 16-byte aligned", i);
    c->w = *w;
    c->have_w = true;
    return pack_weights(c);
}

extern "C" int32_t vuib_codec_enc_check_flag(VuibCodecEnc* c, void* stream) {
    if (!c) return VUIB_ERR_NULL;
    if (!c->packed) return fail(c, VUIB_ERR_UNBOUND, "encoder workspace or weights not bound");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int flag = 0;
    CK(cudaMemcpyAsync(&flag, c->ws + c->off_flag, sizeof(int), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    if (!flag) return VUIB_OK;
    CK(cudaMemsetAsync(c->ws + c->off_flag, 0, sizeof(int), s));
    CK(cudaStreamSynchronize(s));
    return fail(c, VUIB_ERR_DEVICE_FLAG, "encoder device flag 0x%x: a bounded wait inside a kernel ran out", flag);
}

extern "C" int32_t vuib_codec_enc_read_latent(VuibCodecEnc* c, float* out_host, int32_t n, void* stream) {
    if (!c || !out_host) return VUIB_ERR_NULL;
    if (!c->have_ws) return fail(c, VUIB_ERR_UNBOUND, "encoder workspace not bound");
    if (n < 1 || n > 512 * c->last_frames) return fail(c, VUIB_ERR_RANGE, "latent holds %d floats", 512 * c->last_frames);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int T = c->last_frames;
    float* tmp = new (std::nothrow) float[(size_t)512 * T];   // [128][T][4] on the device
    if (!tmp) return fail(c, VUIB_ERR_CUDA, "out of host memory");
    cudaError_t e = cudaMemcpyAsync(tmp, c->ws + c->off_d, (size_t)512 * T * 4, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    for (int i = 0; e == cudaSuccess && i < n; ++i) {
        const int ch = i / T, t = i % T;
        out_host[i] = tmp[((size_t)(ch / 4) * T + t) * 4 + ch % 4];
    }
    delete[] tmp;
    CK(e);
    return VUIB_OK;
}

extern "C" int32_t vuib_codec_enc_encode(VuibCodecEnc* c, const float* audio_dev, int32_t n_samples, int32_t n_q,
                                         int64_t* codes_out_dev, void* stream) {
    if (!c || !audio_dev || !codes_out_dev) return VUIB_ERR_NULL;
    if (!c->packed) return fail(c, VUIB_ERR_UNBOUND, "encoder workspace or weights not bound");
    if (n_samples < 1920 || n_samples % 1920 || n_samples > c->cfg.max_samples)
        return fail(c, VUIB_ERR_RANGE, "n_samples = %d: need a multiple of 1920 up to %d", n_samples, c->cfg.max_samples);
    if (n_q < 1 || n_q > 16) return fail(c, VUIB_ERR_RANGE, "n_q = %d outside [1, 16]", n_q);
    const VuibCodecEncConfig& g = c->cfg;
    const VuibCodecEncWeights& w = c->u;
    if (c->num_sms == 0) {
        int dev = 0;
        CK(cudaGetDevice(&dev));
        CK(cudaDeviceGetAttribute(&c->num_sms, cudaDevAttrMultiProcessorCount, dev));
    }
    using namespace vuis;
    const SgCtx x = {reinterpret_cast<int*>(c->ws + c->off_flag), c->num_sms, true, static_cast<cudaStream_t>(stream), &c->launches};
    auto f32 = [&](size_t off) { return reinterpret_cast<float*>(c->ws + off); };
    auto planes = [&](size_t off, int C, int T) { return sg_planes(c->ws + off, C, T, PAD); };
    auto out = [&](const float* bias, int Cout, int act, SgPlanes o, int div) {
        SgOut e = {};
        e.bias = bias; e.Cout = Cout; e.act = act; e.o = o; e.p_div = div; e.up = 1;
        return e;
    };
    const SgPlanes none = {};
    float* y = f32(c->off_y);
    int T = n_samples, C = g.base_dim;
    // ---- ConvEncoder (qwen_codec.py:293-311)
    {
        EInArgs a = {audio_dev, w.conv_in.w, w.conv_in.b, y, planes(c->off_p[0], C, T), T};
        CK(sg_run(x, k_ein, dim3((T + 127) / 128), dim3(256), 0, a));
    }
    for (int i = 0; i < 4; ++i) {
        const int r = g.ratios[i];
        const SgPlanes in = planes(c->off_p[0], C, T), mid = planes(c->off_p[1], C / 2, T), str = planes(c->off_p[2], C * r, T / r);
        // ResBlock: y + conv1(ELU(conv3(ELU(y)))), kept only as ELU(...) in the order in which the strided convolution reads it
        CK(sg_launch(x, c->pk.c3[i], in, T, 1, out(w.res[i].c3.b, C / 2, SA_ELU, mid, 1)));
        SgOut o = out(w.res[i].c1.b, C, SA_ELU, str, r);
        o.res = y;
        o.y_rows = T;
        CK(sg_launch(x, c->pk.c1[i], mid, T, 1, o));
        T /= r;
        C *= 2;
        o = out(w.down[i].b, C, SA_ELU, planes(c->off_p[0], C, T), 1);
        o.y = i < 3 ? y : nullptr;
        o.y_rows = T;
        CK(sg_launch(x, c->pk.down[i], str, T, 1, o));
    }
    const int D = g.d_model, H = g.n_heads;
    float* xr = f32(c->off_x);
    {
        SgOut o = out(w.conv_out.b, D, SA_NONE, none, 1);
        o.y = xr;
        o.y_rows = T;
        CK(sg_launch(x, c->pk.out, planes(c->off_p[0], C, T), T, 1, o));
    }
    // ---- EncTransformer (314-365) on 25 Hz frames
    float* q = f32(c->off_q);
    const SgPlanes xp = planes(c->off_xp, D, T), gp = planes(c->off_gp, g.mlp_dim, T), half = planes(c->off_xp, 2 * D, T / 2);
    for (int l = 0; l < g.n_layers; ++l) {
        const VuibEncLayerW& lw = w.layer[l];
        SNormArgs na = {xr, T, lw.ln1_w, lw.ln1_b, nullptr, nullptr, 1e-5f, xp, T};
        CK(sg_run(x, k_snorm<SN_LAYER, 512>, dim3((T + 7) / 8), dim3(256), 0, na));
        SgOut o = out(nullptr, 3 * D, SA_NONE, none, 1);
        o.y = q;
        o.y_rows = T;
        CK(sg_launch(x, c->pk.wqkv[l], xp, T, 1, o));
        SAttnArgs aa = {q, T, f32(c->off_rope), g.max_samples / 960, xp, T, H};
        CK(sat_launch(x, aa));
        o = out(nullptr, D, SA_NONE, none, 1);
        o.res = o.y = xr;
        o.scale = lw.attn_scale;
        o.y_rows = T;
        CK(sg_launch(x, c->pk.wo[l], xp, T, 1, o));
        na.w = lw.ln2_w;
        na.b = lw.ln2_b;
        CK(sg_run(x, k_snorm<SN_LAYER, 512>, dim3((T + 7) / 8), dim3(256), 0, na));
        CK(sg_launch(x, c->pk.fc1[l], xp, T, 1, out(nullptr, g.mlp_dim, SA_GELU, gp, 1)));
        o = out(nullptr, D, SA_NONE, l == g.n_layers - 1 ? half : none, 2);   // the last layer's output feeds the stride-2 convolution
        o.res = o.y = xr;
        o.scale = lw.mlp_scale;
        o.y_rows = T;
        CK(sg_launch(x, c->pk.fc2[l], gp, T, 1, o));
    }
    // ---- downsample to 12.5 Hz, project, quantise
    T /= 2;
    c->last_frames = T;
    const SgPlanes dp = planes(c->off_dp, D, T);
    SgOut o = out(nullptr, D, SA_NONE, dp, 1);
    o.y = f32(c->off_d);
    o.y_rows = T;
    CK(sg_launch(x, c->pk.half, half, T, 1, o));
    o = out(nullptr, 512, SA_NONE, none, 1);
    o.y = f32(c->off_h);
    o.y_rows = T;
    CK(sg_launch(x, c->pk.books, dp, T, 1, o));
    ERvqArgs r = {};
    r.h = f32(c->off_h);
    r.codes = reinterpret_cast<long long*>(codes_out_dev);
    r.T = T;
    r.n_q = n_q;
    r.flag = x.flag;
    for (int i = 0; i < n_q; ++i) { r.table[i] = w.codebook[i]; r.norm2[i] = w.codebook_norm2[i]; }
    {
        static thread_local int ready = -1;   // device whose copy of the kernel this thread has opted into its shared memory
        int dev = 0;
        CK(cudaGetDevice(&dev));
        if (ready != dev) {
            CK(cudaFuncSetAttribute(k_ervq<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, RV_SMEM));
            CK(cudaFuncSetAttribute(k_ervq<9>, cudaFuncAttributeMaxDynamicSharedMemorySize, RV_SMEM));
        }
        ready = dev;
    }
    const auto waves = [&](int f) { return ((T + f - 1) / f + RV_RESIDENT - 1) / RV_RESIDENT; };
    const int F = waves(9) < waves(8) ? 9 : 8;   // frames of a cluster, see k_ervq
    CK(sg_run(x, F == 9 ? k_ervq<9> : k_ervq<8>, dim3((T + F - 1) / F * RV_CL, 2), dim3(32 * RV_WARPS), RV_SMEM, r));
    return VUIB_OK;
}
