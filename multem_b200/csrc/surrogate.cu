// Kernels of the learned phonon-convergence surrogate: a small convolutional network that maps a
// HAADF image averaged over a few frozen-phonon configurations to the image averaged over many.
//
// Tensors are NCHW. Activations and weights are stored in BF16, every product is accumulated in
// FP32, biases and gradients are FP32, and the optimiser keeps FP32 master weights. Convolutions
// are 3x3 with zero padding 1 ("same" size):
//   forward      out[b,o,y,x]   = bias[o] + sum_{i,ky,kx} w[o,i,ky,kx] * in[b,i,y+ky-1,x+kx-1]
//   data grad    din[b,i,y,x]   = sum_{o,ky,kx} w[o,i,ky,kx] * dout'[b,o,y-ky+1,x-kx+1]
//   weight grad  dw[o,i,ky,kx]  = sum_{b,y,x} dout'[b,o,y,x] * in[b,i,y+ky-1,x+kx-1]
// where dout' is the output gradient masked by the ReLU of the output when the layer has one.
//
// The three convolutions run on the tensor cores as implicit GEMMs (conv_umma.cuh): forward and data
// gradient in one kernel each, the weight gradient as partial sums per pixel range that a second
// kernel adds in order (fixed-order reductions: deterministic results).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>

#include "common.hpp"
#include "conv_umma.cuh"
#include "devmem.hpp"
#include "multem_b200_surrogate.h"

namespace {

__device__ __forceinline__ float bf(const __nv_bfloat16 v) { return __bfloat162float(v); }

// Loss of the two-channel head in units of a per-item scale s_b (the item's noise level; 1 when
// no scales are given). Channel 0 is a correction r to the input image x (prediction
// yh = x + s_b * r), channel 1 an estimate e of |yh - t| / s_b per pixel. Per pixel, with
// dn = (yh - t) / s_b:
//   loss = dn^2 + lambda * (e - |dn|)^2   (the error target is not differentiated)
// gradients (scaled by 1/n) go to dhead as BF16; per-pixel losses to `terms` for a fixed-order sum.
__global__ void surrogate_loss_kernel(const float* head, const __nv_bfloat16* x,
                                      const float* t, const float* scale,
                                      __nv_bfloat16* dhead, float* terms, int B, int HW,
                                      float lambda) {
    mtb::previous_done();
    mtb::next_may_start();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= B * HW) return;
    const int b = p / HW, q = p % HW;
    const float sc = scale ? scale[b] : 1.0f;
    const float r = head[(size_t)b * 2 * HW + q], e = head[(size_t)b * 2 * HW + HW + q];
    const float yh = __fmaf_rn(sc, r, bf(x[p]));
    const float dn = __fdiv_rn(yh - t[p], sc);
    const float ad = fabsf(dn);
    const float n = (float)(B * HW);
    dhead[(size_t)b * 2 * HW + q] = __float2bfloat16_rn(2.0f * dn / n);
    dhead[(size_t)b * 2 * HW + HW + q] = __float2bfloat16_rn(2.0f * lambda * (e - ad) / n);
    terms[p] = dn * dn + lambda * (e - ad) * (e - ad);
}

// Adam step on FP32 master weights; writes the BF16 copy the kernels read.
__global__ void adam_kernel(float* wm, __nv_bfloat16* wb, const float* g,
                            float* m, float* v, int n, float lr, float b1, float b2, float eps,
                            float c1, float c2) {
    mtb::previous_done();
    mtb::next_may_start();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float w = wm[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    wm[i] = w;
    if (wb) wb[i] = __float2bfloat16_rn(w);
}

// 2 x 2 block sum times `scale` ([B*C, H, W] -> [B*C, H/2, W/2]): average pooling with scale 1/4,
// the gradient of nearest-neighbour upsampling with scale 1.
__global__ void pool2_kernel(const __nv_bfloat16* in, __nv_bfloat16* out, int planes, int H,
                             int W, float scale) {
    mtb::previous_done();
    mtb::next_may_start();
    const int Ho = H / 2, Wo = W / 2;
    const size_t n = (size_t)planes * Ho * Wo;
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
        const size_t pl = k / ((size_t)Ho * Wo);
        const int r = (int)(k % ((size_t)Ho * Wo)), y = r / Wo, x = r % Wo;
        const __nv_bfloat16* s = in + (pl * H + 2 * y) * W + 2 * x;
        const float v = (bf(s[0]) + bf(s[1])) + (bf(s[W]) + bf(s[W + 1]));
        out[k] = __float2bfloat16_rn(v * scale);
    }
}

// Nearest-neighbour 2x upsampling times `scale` ([B*C, H, W] -> [B*C, 2H, 2W]): upsampling with
// scale 1, the gradient of average pooling with scale 1/4.
__global__ void upsample2_kernel(const __nv_bfloat16* in, __nv_bfloat16* out, int planes,
                                 int H, int W, float scale) {
    mtb::previous_done();
    mtb::next_may_start();
    const int Ho = 2 * H, Wo = 2 * W;
    const size_t n = (size_t)planes * Ho * Wo;
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
        const size_t pl = k / ((size_t)Ho * Wo);
        const int r = (int)(k % ((size_t)Ho * Wo)), y = r / Wo, x = r % Wo;
        out[k] = __float2bfloat16_rn(bf(in[(pl * H + y / 2) * W + x / 2]) * scale);
    }
}

__global__ void add_kernel(const __nv_bfloat16* a, const __nv_bfloat16* b,
                           __nv_bfloat16* out, size_t n) {
    mtb::previous_done();
    mtb::next_may_start();
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x)
        out[k] = __float2bfloat16_rn(bf(a[k]) + bf(b[k]));
}

unsigned elem_grid(size_t n) { return (unsigned)std::min<size_t>((n + 255) / 256, 148 * 16); }

__global__ void to_bf16_kernel(const float* __restrict__ a, __nv_bfloat16* __restrict__ b, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) b[i] = __float2bfloat16_rn(a[i]);
}

template <class F>
mt_status run(F f) {
    try {
        f();
        return MT_OK;
    } catch (const mtb::Error& e) {
        return e.status;
    } catch (...) {
        return MT_ERR_INTERNAL;
    }
}

void check_shape(int B, int Cin, int Cout, int H, int W) {
    if (B <= 0 || Cin <= 0 || Cout <= 0 || H <= 0 || W <= 0 || (size_t)B * H * W > (1u << 30))
        mtb::fail(MT_ERR_INVALID_ARG, "bad convolution shape");
}

// Shared memory that the convolution kernels may ask for: the same limit in every launch, since it is the
// kernel's and other host threads launch it with tiles of another size (227 KB less the static variables).
constexpr int kSmemMax = 232448 - 1024;

constexpr long long kWaitNs = 1000000000ll;  // bound of every wait for the tensor cores (1 s)

// whether every row of w [..][Cin][3][3] (bf16) starts on a 16-byte boundary
int weights_aligned(const void* w, int Cin) { return Cin % 8 == 0 && reinterpret_cast<uintptr_t>(w) % 16 == 0; }

size_t align256(size_t v) { return (v + 255) / 256 * 256; }

// Per-device workspace of the weight gradients (partial sums), grown on demand from the library's
// pool, and the error flag of the convolutions' bounded waits. Calls on one device share them, so
// they must be issued on one stream (or otherwise ordered), as the surrogate's host code does.
struct Workspace {
    unsigned char* p = nullptr;
    size_t bytes = 0;
    int* err = nullptr;
    int dev = 0;
};
std::mutex g_ws_mu;
std::map<int, Workspace> g_ws;

Workspace& workspace(size_t bytes) {
    int dev = 0;
    MTB_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(g_ws_mu);
    Workspace& w = g_ws[dev];
    if (!w.err) {
        w.err = static_cast<int*>(mtb::dev_alloc(256, &w.dev));
        MTB_CUDA(cudaMemset(w.err, 0, sizeof(int)));
    }
    if (w.bytes < bytes) {
        const size_t nb = std::max(bytes, 2 * w.bytes);  // grow geometrically
        if (w.p) mtb::dev_free(w.p, w.dev);  // waits for the device: earlier calls may still use it
        w.p = nullptr;
        w.bytes = 0;
        w.p = static_cast<unsigned char*>(mtb::dev_alloc(nb, &w.dev));
        w.bytes = nb;
    }
    return w;
}

template <int BN, int MT, bool DGRAD>
void conv_launch(const mtb::conv::ConvArgs& a, cudaStream_t st) {
    using T = mtb::conv::ConvTile<BN, MT>;
    auto kern = mtb::conv::conv_kernel<BN, MT, DGRAD>;
    const size_t smem = T::smem(a.im.W, a.Cin, a.ksplit);
    MTB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)((a.im.total() + T::TM - 1) / T::TM), (unsigned)((a.Cout + BN - 1) / BN), (unsigned)a.ksplit);
    cfg.blockDim = dim3(mtb::conv::THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2] = {};
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = (unsigned)a.ksplit;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // as mtb::launch_early
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    MTB_CUDA(cudaLaunchKernelEx(&cfg, kern, a));
}

// How a convolution is cut. The widest tile (up to 64 output channels: more would leave room for one CTA per SM
// only) that, with the input channels shared over up to 8 CTAs, still gives every SM a CTA; two pixel tiles per
// CTA where there are CTAs to spare.
struct ConvPlan {
    int bn, ksplit, blocks;  // output channels per CTA, CTAs that share the input channels, K blocks of each
    bool two;                // pixel tiles per CTA
};
ConvPlan conv_plan(const mtb::conv::Image& im, int Cin, int Cout) {
    const long long tiles = (im.total() + 127) / 128;
    const int nkb = (Cin + mtb::conv::KC - 1) / mtb::conv::KC;
    int most = 1;
    while (most < 8 && 2 * most <= nkb) most *= 2;
    auto ctas = [&](int bn) { return tiles * ((Cout + bn - 1) / bn); };
    ConvPlan p{Cout <= 16 ? 16 : Cout <= 32 ? 32 : 64, 1, nkb, false};
    while (p.bn > 16 && ctas(p.bn) * most < 148) p.bn /= 2;
    // K is cut into `parts` at least (over CTAs and accumulators) where that leaves more than two blocks to each CTA
    const long long m = ((long long)im.B * im.H * im.W + 127) / 128 * ((Cout + 255) / 256);
    const long long parts = (295 + m) / m;
    while (p.ksplit < most && (ctas(p.bn) * p.ksplit < 148 || p.blocks > std::max<long long>(2, 4 * nkb / parts))) {
        p.ksplit *= 2;
        p.blocks = (nkb + p.ksplit - 1) / p.ksplit;
    }
    p.two = ctas(p.bn) >= 4 * 148 && parts == 1;
    return p;
}

template <bool DGRAD>
void conv(mtb::conv::ConvArgs a, cudaStream_t st) {
    const ConvPlan p = conv_plan(a.im, a.Cin, a.Cout);
    a.ksplit = p.ksplit;
    switch (p.bn) {
        case 16: p.two ? conv_launch<16, 2, DGRAD>(a, st) : conv_launch<16, 1, DGRAD>(a, st); break;
        case 32: p.two ? conv_launch<32, 2, DGRAD>(a, st) : conv_launch<32, 1, DGRAD>(a, st); break;
        default: p.two ? conv_launch<64, 2, DGRAD>(a, st) : conv_launch<64, 1, DGRAD>(a, st); break;
    }
}

// How a weight gradient is cut: input channels per CTA (the gradient tile is gathered once for each, so as many as
// the layer has and two stages of shared memory hold) and K blocks per split, for two CTAs per SM (one
// where the tile's tensor memory allows no more).
struct WgradPlan {
    int ni, itiles, otiles, nblk, blk_per_split, splits;
};
WgradPlan wgrad_plan(const mtb::conv::Image& im, int Cin, int Cout) {
    WgradPlan p{};
    p.ni = Cin <= 16 ? 16 : Cin <= 32 ? 32 : Cin <= 64 || mtb::conv::WgradTile<128>::smem(im.W) > (size_t)kSmemMax ? 64 : 128;
    p.itiles = (Cin + p.ni - 1) / p.ni;
    p.otiles = (Cout + mtb::conv::WG_OC - 1) / mtb::conv::WG_OC;
    p.nblk = (int)((im.total() + mtb::conv::WG_PIX - 1) / mtb::conv::WG_PIX);
    const long long tiles = (long long)p.itiles * p.otiles, want = ((p.ni > 64 ? 148 : 296) + tiles - 1) / tiles;
    p.blk_per_split = (int)std::max<long long>(1, (p.nblk + want - 1) / want);
    p.splits = (p.nblk + p.blk_per_split - 1) / p.blk_per_split;
    return p;
}

template <int NI>
void wgrad_launch(mtb::conv::WgradArgs a, const WgradPlan& p, float* dw, float* db, cudaStream_t st) {
    using T = mtb::conv::WgradTile<NI>;
    const int C32 = p.otiles * mtb::conv::WG_OC;
    a.nblk = p.nblk;
    a.blk_per_split = p.blk_per_split;
    const size_t off_b = align256((size_t)p.splits * 9 * a.Cin * C32 * sizeof(float));
    const size_t off_s = off_b + align256((size_t)p.splits * C32 * sizeof(float));
    Workspace& ws = workspace(off_s + (size_t)p.splits * ((a.Cin + 31) / 32) * sizeof(unsigned));
    a.part = reinterpret_cast<float*>(ws.p);
    a.bpart = reinterpret_cast<float*>(ws.p + off_b);
    a.special = reinterpret_cast<unsigned*>(ws.p + off_s);
    a.err = ws.err;
    auto kern = mtb::conv::wgrad_kernel<NI>;
    const size_t smem = T::smem(a.im.W);
    MTB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax));
    mtb::launch_early(true, kern, dim3((unsigned)p.splits, (unsigned)p.itiles, (unsigned)p.otiles), mtb::conv::THREADS, smem, st, a);
    mtb::launch_early(true, mtb::conv::wgrad_finalize_kernel, dim3((unsigned)p.otiles, (unsigned)(a.Cin + 1), 3), 256, 0, st, a,
                      p.splits, dw, db);
}

}  // namespace

extern "C" {

mt_status mt_sg_conv3x3_forward(const void* in, const void* w, const float* bias, void* out_bf16, float* out_f32,
                                int B, int Cin, int Cout, int H, int W, int relu, void* stream) {
    return run([&] {
        check_shape(B, Cin, Cout, H, W);
        if (!in || !w || (!out_bf16 && !out_f32)) mtb::fail(MT_ERR_INVALID_ARG, "NULL tensor");
        conv<false>({(const __nv_bfloat16*)in, nullptr, (const __nv_bfloat16*)w, bias, (__nv_bfloat16*)out_bf16, out_f32,
                     mtb::conv::image(B, H, W), Cin, Cout, relu, weights_aligned(w, Cin), 1, workspace(0).err, kWaitNs}, (cudaStream_t)stream);
    });
}

mt_status mt_sg_conv3x3_backward_data(const void* dout, const void* out_mask, const void* w, void* din, int B, int Cin,
                                      int Cout, int H, int W, void* stream) {
    return run([&] {
        check_shape(B, Cin, Cout, H, W);
        if (!dout || !w || !din) mtb::fail(MT_ERR_INVALID_ARG, "NULL tensor");
        // the data gradient is a convolution of the masked output gradient (Cout channels) with the
        // flipped, transposed kernel
        conv<true>({(const __nv_bfloat16*)dout, (const __nv_bfloat16*)out_mask, (const __nv_bfloat16*)w, nullptr,
                    (__nv_bfloat16*)din, nullptr, mtb::conv::image(B, H, W), Cout, Cin, 0, weights_aligned(w, Cin), 1, workspace(0).err,
                    kWaitNs}, (cudaStream_t)stream);
    });
}

mt_status mt_sg_conv3x3_backward_weight(const void* in, const void* dout, const void* out_mask, float* dw, float* db,
                                        int B, int Cin, int Cout, int H, int W, void* stream) {
    return run([&] {
        check_shape(B, Cin, Cout, H, W);
        if (!in || !dout || !dw || !db) mtb::fail(MT_ERR_INVALID_ARG, "NULL tensor");
        const cudaStream_t st = (cudaStream_t)stream;
        mtb::conv::WgradArgs a{};
        a.in = (const __nv_bfloat16*)in;
        a.dout = (const __nv_bfloat16*)dout;
        a.mask = (const __nv_bfloat16*)out_mask;
        a.im = mtb::conv::image(B, H, W);
        a.Cin = Cin;
        a.Cout = Cout;
        a.wait_ns = kWaitNs;
        const WgradPlan p = wgrad_plan(a.im, Cin, Cout);
        switch (p.ni) {
            case 16: wgrad_launch<16>(a, p, dw, db, st); break;
            case 32: wgrad_launch<32>(a, p, dw, db, st); break;
            case 64: wgrad_launch<64>(a, p, dw, db, st); break;
            default: wgrad_launch<128>(a, p, dw, db, st); break;
        }
    });
}

mt_status mt_sg_conv3x3_plan(int B, int Cin, int Cout, int H, int W, int pass, int* plan) {
    return run([&] {
        check_shape(B, Cin, Cout, H, W);
        if (pass < 0 || pass > 2 || !plan) mtb::fail(MT_ERR_INVALID_ARG, "bad plan arguments");
        const mtb::conv::Image im = mtb::conv::image(B, H, W);
        if (pass == 2) {
            const WgradPlan p = wgrad_plan(im, Cin, Cout);
            const int v[5] = {p.ni, 1, p.splits, p.blk_per_split, mtb::conv::WgradTile<16>::seg(W) != W + 1};
            std::copy(v, v + 5, plan);
        } else {
            const ConvPlan p = pass ? conv_plan(im, Cout, Cin) : conv_plan(im, Cin, Cout);
            const int seg = p.two ? mtb::conv::ConvTile<16, 2>::seg(W) : mtb::conv::ConvTile<16, 1>::seg(W);
            const int v[5] = {p.bn, p.two ? 2 : 1, p.ksplit, p.blocks, seg != W + 1};
            std::copy(v, v + 5, plan);
        }
    });
}

mt_status mt_sg_check(void* stream) {
    return run([&] {
        MTB_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
        int dev = 0;
        MTB_CUDA(cudaGetDevice(&dev));
        int* err = nullptr;
        {
            std::lock_guard<std::mutex> lk(g_ws_mu);
            auto it = g_ws.find(dev);
            if (it != g_ws.end()) err = it->second.err;
        }
        if (!err) return;
        int e = 0;
        MTB_CUDA(cudaMemcpy(&e, err, sizeof(int), cudaMemcpyDeviceToHost));
        if (e) {
            MTB_CUDA(cudaMemset(err, 0, sizeof(int)));
            mtb::fail(MT_ERR_TIMEOUT, "a convolution gave up waiting for the tensor cores");
        }
    });
}

mt_status mt_sg_loss(const float* head, const void* x, const float* target, const float* scale, void* dhead,
                     float* terms, int B, int H, int W, float lambda, void* stream) {
    return run([&] {
        check_shape(B, 1, 2, H, W);
        if (!head || !x || !target || !dhead || !terms) mtb::fail(MT_ERR_INVALID_ARG, "NULL tensor");
        const int n = B * H * W;
        mtb::launch_early(true, surrogate_loss_kernel, (n + 255) / 256, 256, 0, (cudaStream_t)stream, head, (const __nv_bfloat16*)x,
                          target, scale, (__nv_bfloat16*)dhead, terms, B, H * W, lambda);
    });
}

mt_status mt_sg_adam(float* w, void* w_bf16, const float* g, float* m, float* v, int n, float lr, float b1, float b2,
                     float eps, int step, void* stream) {
    return run([&] {
        if (n <= 0 || step <= 0) mtb::fail(MT_ERR_INVALID_ARG, "bad Adam arguments");
        const float c1 = 1.0f - std::pow(b1, (float)step), c2 = 1.0f - std::pow(b2, (float)step);
        mtb::launch_early(true, adam_kernel, (n + 255) / 256, 256, 0, (cudaStream_t)stream, w, (__nv_bfloat16*)w_bf16, g, m, v, n,
                          lr, b1, b2, eps, c1, c2);
    });
}

mt_status mt_sg_pool2(const void* in, void* out, int B, int C, int H, int W, float scale, void* stream) {
    return run([&] {
        check_shape(B, C, 1, H, W);
        if (H % 2 || W % 2) mtb::fail(MT_ERR_INVALID_ARG, "pooling needs even H and W");
        if (!in || !out) mtb::fail(MT_ERR_INVALID_ARG, "NULL tensor");
        const size_t n = (size_t)B * C * (H / 2) * (W / 2);
        mtb::launch_early(true, pool2_kernel, elem_grid(n), 256, 0, (cudaStream_t)stream, (const __nv_bfloat16*)in,
                          (__nv_bfloat16*)out, B * C, H, W, scale);
    });
}

mt_status mt_sg_upsample2(const void* in, void* out, int B, int C, int H, int W, float scale, void* stream) {
    return run([&] {
        check_shape(B, C, 1, 2 * H, 2 * W);
        if (!in || !out) mtb::fail(MT_ERR_INVALID_ARG, "NULL tensor");
        const size_t n = (size_t)B * C * (2 * H) * (2 * W);
        mtb::launch_early(true, upsample2_kernel, elem_grid(n), 256, 0, (cudaStream_t)stream, (const __nv_bfloat16*)in,
                          (__nv_bfloat16*)out, B * C, H, W, scale);
    });
}

mt_status mt_sg_add(const void* a, const void* b, void* out, long long n, void* stream) {
    return run([&] {
        if (n < 0 || (n > 0 && (!a || !b || !out))) mtb::fail(MT_ERR_INVALID_ARG, "bad add arguments");
        if (n == 0) return;
        mtb::launch_early(true, add_kernel, elem_grid((size_t)n), 256, 0, (cudaStream_t)stream, (const __nv_bfloat16*)a,
                          (const __nv_bfloat16*)b, (__nv_bfloat16*)out, (size_t)n);
    });
}

mt_status mt_sg_to_bf16(const float* a, void* b, int n, void* stream) {
    return run([&] {
        if (n <= 0) return;
        to_bf16_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(a, (__nv_bfloat16*)b, n);
        MTB_CUDA(cudaGetLastError());
    });
}

}  // extern "C"
