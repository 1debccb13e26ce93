"""Kernels of the learned surrogate (include/multem_b200_surrogate.h) against a PyTorch FP32
reference of the same operations on the same BF16-rounded values, the whole encoder-decoder's
gradients against PyTorch CPU autograd, and a short training run.

Bounds: forward and data gradient 1e-5 relative (FP32 sums of the same products in a different
order), weight gradient 1e-4 (long sums over the batch and image)."""
import ctypes as C

import numpy as np
import pytest

from multem_b200 import capi

pytestmark = pytest.mark.gpu


def _p(t):
    return C.c_void_p(t.data_ptr())


def _rel(a, b):
    return float((a - b).norm() / b.norm())


@pytest.mark.parametrize("B,Cin,Cout,H,W", [(2, 3, 5, 20, 37), (3, 8, 16, 32, 32), (1, 16, 2, 16, 16),
                                             (2, 64, 128, 32, 32), (1, 256, 256, 8, 8), (4, 32, 32, 64, 64),
                                             (3, 128, 64, 16, 24)])
def test_conv3x3_forward_and_gradients_match_torch(B, Cin, Cout, H, W):
    torch = pytest.importorskip("torch")
    F = torch.nn.functional
    lib = capi.load()
    g = torch.Generator().manual_seed(B * 100 + Cin)
    x = torch.randn(B, Cin, H, W, generator=g).to(torch.bfloat16).cuda()
    w = (torch.randn(Cout, Cin, 3, 3, generator=g) * 0.3).to(torch.bfloat16).cuda()
    b = torch.randn(Cout, generator=g).cuda()
    # forward with ReLU, bf16 and fp32 outputs
    yb = torch.empty(B, Cout, H, W, device="cuda", dtype=torch.bfloat16)
    yf = torch.empty(B, Cout, H, W, device="cuda")
    capi.check(lib.mt_sg_conv3x3_forward(_p(x), _p(w), _p(b), _p(yb), _p(yf), B, Cin, Cout, H, W, 1, None))
    torch.cuda.synchronize()
    ref = F.relu(F.conv2d(x.float(), w.float(), b, padding=1))
    assert _rel(yf, ref) < 1e-5
    assert _rel(yb.float(), ref) < 1e-2  # BF16 storage
    # gradients through the ReLU: dout masked where the (bf16) output is not positive
    dout = torch.randn(B, Cout, H, W, generator=g).to(torch.bfloat16).cuda()
    xr = x.float().clone().requires_grad_(True)
    wr = w.float().clone().requires_grad_(True)
    br = b.clone().requires_grad_(True)
    out = F.conv2d(xr, wr, br, padding=1)
    mask = (yb.float() > 0).float()
    out.backward(dout.float() * mask)
    din = torch.empty_like(x)
    capi.check(lib.mt_sg_conv3x3_backward_data(_p(dout), _p(yb), _p(w), _p(din), B, Cin, Cout, H, W, None))
    dw = torch.empty(Cout, Cin, 3, 3, device="cuda")
    db = torch.empty(Cout, device="cuda")
    capi.check(lib.mt_sg_conv3x3_backward_weight(_p(x), _p(dout), _p(yb), _p(dw), _p(db), B, Cin, Cout, H, W, None))
    torch.cuda.synchronize()
    assert _rel(din.float(), xr.grad) < 1e-2  # din stored in BF16
    assert _rel(dw, wr.grad) < 1e-4
    assert _rel(db, br.grad) < 1e-4


# tile edges of the implicit GEMM: rows around the 128- and 256-pixel tiles (one band of pixels or three
# segments), channels that are no multiple of 8, 16 or 32, and clusters that share the input channels unevenly
@pytest.mark.parametrize("B,Cin,Cout,H,W", [(1, 40, 24, 3, 127), (1, 33, 40, 2, 130), (1, 16, 70, 1, 257), (2, 4, 3, 3, 600),
                                             (1, 300, 33, 4, 9), (1, 96, 256, 4, 4), (3, 1, 1, 1, 1), (20, 8, 40, 64, 64),
                                             (20, 9, 2, 64, 63), (20, 40, 32, 63, 64), (2, 130, 64, 5, 129)])
def test_conv3x3_at_tile_edges(B, Cin, Cout, H, W):
    test_conv3x3_forward_and_gradients_match_torch(B, Cin, Cout, H, W)


def test_weight_gradient_with_infinite_and_nan_inputs():
    """An infinity or NaN at an image's edge reaches only the taps whose products it is part of (the
    zeros of the padding times the gradient, never the input times a gradient outside the image)."""
    torch = pytest.importorskip("torch")
    lib = capi.load()
    B, Cin, Cout, H, W = 2, 3, 4, 5, 6
    g = torch.Generator().manual_seed(9)
    x = torch.randn(B, Cin, H, W, generator=g)
    x[0, 0, 0, 0], x[1, 1, H - 1, W - 1] = float("inf"), float("nan")
    d = 1 + torch.rand(B, Cout, H, W, generator=g)
    x, d = x.to(torch.bfloat16), d.to(torch.bfloat16)
    cols = torch.nn.functional.unfold(x.double(), 3, padding=1).reshape(B, Cin, 9, H * W)
    ref = torch.einsum("boq,bctq->oct", d.double().reshape(B, Cout, H * W), cols).reshape(Cout, Cin, 3, 3)
    xd, dd = x.cuda(), d.cuda()
    dw = torch.empty(Cout, Cin, 3, 3, device="cuda")
    db = torch.empty(Cout, device="cuda")
    capi.check(lib.mt_sg_conv3x3_backward_weight(_p(xd), _p(dd), None, _p(dw), _p(db), B, Cin, Cout, H, W, None))
    dw = dw.cpu().double()
    assert torch.equal(dw.isnan(), ref.isnan()) and torch.equal(dw.isinf(), ref.isinf())
    ok = ref.isfinite()
    assert ok.any() and not ok.all()
    assert _rel(dw[ok], ref[ok]) < 1e-4


# how mt_sg_conv3x3_plan cuts each shape: forward, data gradient (channels per CTA, pixel tiles, CTAs per sum, K blocks per
# CTA, segments) and weight gradient. From three blocks per CTA on, a stage of shared memory is used again.
PLANS = {(16, 32, 32, 64, 64): ((32, 1, 1, 1, 0), (32, 1, 1, 1, 0), (32, 1, 265, 2, 0)),
         (8, 256, 64, 64, 64): ((64, 1, 1, 8, 0), (64, 1, 1, 2, 0), (128, 1, 34, 8, 0)),
         (32, 256, 128, 12, 12): ((64, 1, 4, 2, 0), (64, 1, 2, 2, 0), (128, 1, 15, 3, 0)),
         (64, 8, 16, 4, 300): ((16, 2, 1, 1, 1), (16, 2, 1, 1, 1), (16, 1, 251, 3, 1)),
         (16, 160, 64, 64, 64): ((64, 1, 1, 5, 0), (64, 2, 1, 2, 0), (128, 1, 36, 15, 0)),
         (16, 72, 40, 8, 300): ((64, 1, 1, 3, 1), (64, 2, 1, 2, 1), (64, 1, 68, 5, 1)),
         (4, 512, 64, 40, 40): ((64, 1, 4, 4, 0), (64, 1, 1, 2, 0), (128, 1, 18, 3, 0)),
         (1, 800, 16, 24, 24): ((16, 1, 8, 4, 0), (16, 1, 1, 1, 0), (128, 1, 5, 1, 0)),
         (1, 300, 200, 9, 31): ((32, 1, 8, 2, 0), (16, 1, 4, 2, 0), (128, 1, 3, 1, 0)),
         (8, 96, 64, 130, 130): ((64, 2, 1, 3, 0), (64, 2, 1, 2, 0), (64, 1, 72, 15, 1)),
         (5, 36, 64, 100, 260): ((64, 2, 1, 2, 1), (64, 2, 1, 2, 1), (64, 1, 148, 7, 1)),
         (2, 520, 48, 16, 140): ((64, 1, 4, 5, 1), (64, 1, 1, 2, 1), (64, 1, 13, 3, 1)),
         (40, 32, 48, 64, 64): ((64, 2, 1, 1, 0), (32, 2, 1, 2, 0), (32, 1, 147, 9, 0)),
         (30, 100, 20, 64, 64): ((32, 2, 1, 4, 0), (64, 2, 1, 1, 0), (128, 1, 142, 7, 0)),
         (16, 200, 24, 10, 300): ((32, 1, 1, 7, 1), (64, 2, 1, 1, 1), (64, 1, 69, 6, 1))}


@pytest.mark.parametrize("shape", PLANS)
def test_conv3x3_on_every_way_of_cutting(shape):
    """Every tile width with one and two pixel tiles, sums shared by up to eight CTAs, stages used again, bands and segments:
    the plans are those listed, together with their results against torch."""
    lib = capi.load()
    B, Cin, Cout, H, W = shape
    for k, want in enumerate(PLANS[shape]):
        plan = (C.c_int * 5)()
        capi.check(lib.mt_sg_conv3x3_plan(B, Cin, Cout, H, W, k, plan))
        assert tuple(plan) == want, (k, tuple(plan))
    test_conv3x3_forward_and_gradients_match_torch(*shape)


@pytest.mark.parametrize("at", [(0, 0, 0), (0, 0, 5), (0, 4, 0), (1, 0, 0), (1, 4, 5), (1, 2, 3)])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_weight_gradient_with_an_infinite_gradient(value, at):
    """An infinite gradient times the zero beside the image is NaN, at the corners of the first and the last image too."""
    torch = pytest.importorskip("torch")
    lib = capi.load()
    B, Cin, Cout, H, W = 2, 3, 4, 5, 6
    g = torch.Generator().manual_seed(9)
    x = (1 + torch.rand(B, Cin, H, W, generator=g)).to(torch.bfloat16)
    d = torch.randn(B, Cout, H, W, generator=g)
    d[at[0], 2, at[1], at[2]] = value
    d = d.to(torch.bfloat16)
    cols = torch.nn.functional.unfold(x.double(), 3, padding=1).reshape(B, Cin, 9, H * W)
    ref = torch.einsum("boq,bctq->oct", d.double().reshape(B, Cout, H * W), cols).reshape(Cout, Cin, 3, 3)
    xd, dd = x.cuda(), d.cuda()
    dw, db = torch.empty(Cout, Cin, 3, 3, device="cuda"), torch.empty(Cout, device="cuda")
    capi.check(lib.mt_sg_conv3x3_backward_weight(_p(xd), _p(dd), None, _p(dw), _p(db), B, Cin, Cout, H, W, None))
    dw, db = dw.cpu().double(), db.cpu()
    assert torch.equal(dw.isnan(), ref.isnan()) and torch.equal(dw.isinf(), ref.isinf())
    ok = ref.isfinite()
    assert _rel(dw[ok], ref[ok]) < 1e-4
    assert torch.equal(db.isfinite(), torch.tensor([True, True, False, True]))


# infinities and NaN in some channels and splits of a layer of many (296 splits of 8 blocks), and everywhere
@pytest.mark.parametrize("what", ["few", "one channel", "all"])
def test_weight_gradient_with_infinite_and_nan_inputs_of_a_large_layer(what):
    """Only sums that such an input is part of change, and they cost little more: a diverged step of 16 x 32 channels
    at 128 x 128 takes less than ten times a finite one (20 ms, 300 times, where every sum is taken again to its end)."""
    torch = pytest.importorskip("torch")
    lib = capi.load()
    B, C_, H, W = 16, 32, 128, 128
    g = torch.Generator().manual_seed(2)
    x = torch.randn(B, C_, H, W, generator=g)
    d = torch.randn(B, C_, H, W, generator=g).to(torch.bfloat16).cuda()
    finite = x.to(torch.bfloat16).cuda()
    if what == "few":
        x[0, 3, 0, 0], x[7, 3, 64, 127], x[15, 31, 127, 127] = float("inf"), float("-inf"), float("nan")
    elif what == "one channel":
        x[:, 17] = float("nan")
    else:
        x[:] = float("nan")
    xd = x.to(torch.bfloat16).cuda()
    dw, db = torch.empty(C_, C_, 3, 3, device="cuda"), torch.empty(C_, device="cuda")

    def grad(v):
        capi.check(lib.mt_sg_conv3x3_backward_weight(_p(v), _p(d), None, _p(dw), _p(db), B, C_, C_, H, W, None))

    def time_of(v):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        best = 1e9
        for _ in range(5):
            e[0].record()
            grad(v)
            e[1].record()
            torch.cuda.synchronize()
            best = min(best, e[0].elapsed_time(e[1]))
        return best

    grad(finite)
    base = dw.clone()
    grad(xd)
    cols = torch.nn.functional.unfold(xd.double(), 3, padding=1).reshape(B, C_, 9, H * W)
    ref = torch.einsum("boq,bctq->oct", d.double().reshape(B, C_, H * W), cols).reshape(C_, C_, 3, 3)
    assert torch.equal(dw.isnan(), ref.isnan()) and torch.equal(dw.isinf(), ref.isinf())
    touched = (~xd.isfinite()).any(0).any(-1).any(-1)
    assert torch.equal(dw[:, ~touched], base[:, ~touched])
    ok = ref.isfinite()
    if ok.any():
        assert _rel(dw.double()[ok], ref[ok]) < 1e-4
    assert time_of(xd) < 10 * time_of(finite) + 1.0  # ms


def test_loss_and_adam_match_their_formulas():
    torch = pytest.importorskip("torch")
    lib = capi.load()
    B, H, W, lam = 2, 16, 16, 0.5
    g = torch.Generator().manual_seed(3)
    head = torch.randn(B, 2, H, W, generator=g).cuda()
    x = torch.rand(B, 1, H, W, generator=g).to(torch.bfloat16).cuda()
    t = torch.rand(B, 1, H, W, generator=g).cuda()
    dh = torch.empty(B, 2, H, W, device="cuda", dtype=torch.bfloat16)
    terms = torch.empty(B, H, W, device="cuda")
    sc = torch.tensor([1.0, 0.5], device="cuda")
    capi.check(lib.mt_sg_loss(_p(head), _p(x), _p(t), _p(sc), _p(dh), _p(terms), B, H, W, lam, None))
    s = sc[:, None, None]
    d = (x.float()[:, 0] + s * head[:, 0] - t[:, 0]) / s
    e = head[:, 1]
    n = B * H * W
    assert _rel(terms, d * d + lam * (e - d.abs()) ** 2) < 1e-6
    assert _rel(dh.float()[:, 0], 2 * d / n) < 1e-2 and _rel(dh.float()[:, 1], 2 * lam * (e - d.abs()) / n) < 1e-2
    w = torch.randn(100, generator=g).cuda()
    w0 = w.clone()
    gr = torch.randn(100, generator=g).cuda()
    m = torch.zeros(100, device="cuda")
    v = torch.zeros(100, device="cuda")
    capi.check(lib.mt_sg_adam(_p(w), None, _p(gr), _p(m), _p(v), 100, 1e-2, 0.9, 0.999, 1e-8, 1, None))
    torch.cuda.synchronize()
    mh, vh = gr, gr * gr  # first step: bias-corrected moments are the gradient and its square
    assert _rel(w, w0 - 1e-2 * mh / (vh.sqrt() + 1e-8)) < 1e-5


class _RoundBF16:
    """Rounds activations to BF16 in the forward pass (the kernels store them in BF16); gradients
    pass unchanged."""

    @staticmethod
    def apply(x):
        import torch
        return x + (x.to(torch.bfloat16).float() - x).detach()


def _torch_reference(net, x, t, lam):
    """The network of multem_b200.surrogate.Net in PyTorch FP32 autograd on the CPU, on the same
    BF16 weights; returns (head, weight gradients, bias gradients)."""
    import torch
    F = torch.nn.functional
    R = _RoundBF16.apply
    W = [w.float().cpu().requires_grad_(True) for w in net.wb]
    Bs = [b.cpu().requires_grad_(True) for b in net.b]
    x, t = x.cpu(), t.cpu()

    def conv(k, h, relu=True):
        y = F.conv2d(h, W[k], Bs[k], padding=1)
        return R(F.relu(y)) if relu else y

    L = net.L
    enc, h = [], x.float()
    for l in range(L):
        if l > 0:
            h = R(F.avg_pool2d(h, 2))
        h = conv(2 * l + 1, conv(2 * l, h))
        enc.append(h)
    k = 2 * L
    for l in range(L - 2, -1, -1):
        u = F.interpolate(h, scale_factor=2, mode="nearest")
        h = conv(k + 1, R(conv(k, u) + enc[l]))
        k += 2
    head = conv(k, h, relu=False)
    d = x.float()[:, 0] + head[:, 0] - t[:, 0]
    loss = (d * d + lam * (head[:, 1] - d.abs().detach()) ** 2).mean()
    loss.backward()
    return head.detach(), [w.grad for w in W], [b.grad for b in Bs]


def test_encoder_decoder_gradients_match_torch_autograd():
    """Forward and every weight/bias gradient of a 3-level encoder-decoder (pooling, upsampling,
    additive skips, ReLU masks) against PyTorch FP32 autograd. Activations and activation
    gradients are BF16 in the kernels, so the bound is 3e-2 relative L2 per tensor; a wrong index,
    mask or missing skip gradient gives errors of order 1."""
    torch = pytest.importorskip("torch")
    from multem_b200.surrogate import Net
    net = Net(widths=(8, 16, 32), in_ch=2, seed=4)
    for b in net.b:  # non-zero biases so that the ReLU masks matter
        b.copy_(torch.randn(b.shape, generator=torch.Generator().manual_seed(b.numel())).cuda() * 0.1)
    g = torch.Generator().manual_seed(5)
    x = (1 + 0.3 * torch.rand(4, 2, 16, 16, generator=g)).to(torch.bfloat16).cuda()
    t = (1 + 0.3 * torch.rand(4, 1, 16, 16, generator=g)).cuda()
    saved, head = net.forward(x)
    dhead, _ = net.loss_grad(head, x, t, lam=0.5)
    gw, gb = net.backward(saved, dhead)
    torch.cuda.synchronize()
    ref_head, rw, rb = _torch_reference(net, x, t, 0.5)
    head, gw, gb = head.cpu(), [v.cpu() for v in gw], [v.cpu() for v in gb]
    assert _rel(head, ref_head) < 1e-2
    for k in range(len(net.layers)):
        assert _rel(gw[k], rw[k]) < 3e-2, f"weight gradient of conv {k}: {_rel(gw[k], rw[k]):.3e}"
        assert _rel(gb[k], rb[k]) < 3e-2, f"bias gradient of conv {k}: {_rel(gb[k], rb[k]):.3e}"


def test_pool_upsample_add_kernels():
    torch = pytest.importorskip("torch")
    F = torch.nn.functional
    lib = capi.load()
    x = torch.randn(2, 3, 8, 12, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()
    y = torch.empty(2, 3, 4, 6, device="cuda", dtype=torch.bfloat16)
    capi.check(lib.mt_sg_pool2(_p(x), _p(y), 2, 3, 8, 12, 0.25, None))
    u = torch.empty(2, 3, 16, 24, device="cuda", dtype=torch.bfloat16)
    capi.check(lib.mt_sg_upsample2(_p(x), _p(u), 2, 3, 8, 12, 1.0, None))
    z = torch.empty_like(x)
    capi.check(lib.mt_sg_add(_p(x), _p(x), _p(z), x.numel(), None))
    torch.cuda.synchronize()
    assert _rel(y.float(), F.avg_pool2d(x.float(), 2)) < 4e-3
    assert torch.equal(u.float(), F.interpolate(x.float(), scale_factor=2, mode="nearest"))
    assert torch.equal(z.float(), 2 * x.float())
    assert lib.mt_sg_pool2(_p(x), _p(y), 2, 3, 7, 12, 0.25, None) != 0  # odd height refused


def test_training_reduces_the_loss():
    """A few hundred steps on synthetic data (noisy copies of smooth images) cut the loss."""
    torch = pytest.importorskip("torch")
    from multem_b200.surrogate import Net
    rng = np.random.default_rng(0)
    yy, xx = np.mgrid[0:32, 0:32] / 32.0
    clean = np.stack([1 + 0.5 * np.cos(2 * np.pi * (k % 3 + 1) * xx) * np.cos(2 * np.pi * (k % 2 + 1) * yy)
                      for k in range(64)])
    noisy = clean * (1 + 0.05 * rng.standard_normal(clean.shape))
    X = torch.from_numpy(noisy[:, None].astype(np.float32)).cuda().to(torch.bfloat16)
    T = torch.from_numpy(clean[:, None].astype(np.float32)).cuda()
    net = Net(widths=(16, 32), in_ch=1)
    first = np.mean([net.train_step(X, T, lr=2e-3) for _ in range(5)])
    for _ in range(300):
        last = net.train_step(X, T, lr=2e-3)
    assert last < 0.5 * first


def test_trained_surrogate_gains_over_the_plain_few_configuration_image():
    """What the committed network gains over the method without it, on a specimen outside its
    training, calibration and evaluation sets (fcc Au(001), 16 nm, beam tilted 1.7 deg, 32 x 32
    HAADF raster over 2 x 2 cells, 64 phonon configurations): its estimate from the first 4
    configurations is closer to the 64-configuration image than the plain 4-configuration mean,
    with and without the lattice fold, and so is the folded estimate from 16 configurations; an
    estimate the gate accepts is within twice the gate of the 64-configuration image."""
    pytest.importorskip("torch")
    from multem_b200 import surrogate as S
    sg = S.Surrogate.load()
    im, _ = S.per_configuration_images(S.haadf_specimen(101))
    full = im.mean(axis=0)
    cases = [(4, S.PERIOD), (4, None), (16, S.PERIOD)]
    for n, period in cases:
        small = im[:n].mean(axis=0)
        pred, est, ok = sg.predict(small, n, period)
        e_plain, e_learned = S.rel_rms(small, full), S.rel_rms(pred, full)
        print(f"n={n} fold={bool(period)}: plain {e_plain:.4f} learned {e_learned:.4f} estimate {est:.4f} accepted {ok}")
        assert e_learned < e_plain
        if ok:
            assert e_learned <= 2 * sg.gate


# An accumulator of the tensor core loses up to about 1.5e-8 of the sum per product of 16 that it takes in (measured
# 1.1e-8); small batches spread theirs over four accumulators and, where there are many channels, over CTAs. n: products
# in a row (a K block of 32 channels gives each accumulator 5 at most); 5e-8 for the FP32 sum and result.
@pytest.mark.parametrize("B,Cin,Cout,H,W,n", [(32, 32, 32, 32, 32, 5), (32, 32, 64, 16, 16, 5), (32, 64, 32, 32, 32, 10),
                                               (1, 256, 256, 8, 8, 5), (32, 256, 128, 8, 8, 10), (8, 256, 64, 64, 64, 40),
                                               (16, 32, 32, 128, 128, 18)])
def test_convolution_sums_against_64_bits(B, Cin, Cout, H, W, n):
    torch = pytest.importorskip("torch")
    lib = capi.load()
    g = torch.Generator().manual_seed(Cin)
    x = torch.randn(B, Cin, H, W, generator=g).to(torch.bfloat16).cuda()
    w = (torch.randn(Cout, Cin, 3, 3, generator=g) * (2 / (9 * Cin)) ** 0.5).to(torch.bfloat16).cuda()
    y = torch.empty(B, Cout, H, W, device="cuda")
    capi.check(lib.mt_sg_conv3x3_forward(_p(x), _p(w), None, None, _p(y), B, Cin, Cout, H, W, 0, None))
    ref = torch.nn.functional.conv2d(x.double(), w.double(), padding=1)
    assert _rel(y.double(), ref) < 1.5e-8 * n + 5e-8
