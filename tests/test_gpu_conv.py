"""Learned-denoiser kernels against plain PyTorch fp32 references on the
same bf16-rounded operands: 3x3 convolution forward, input gradient and
weight / bias gradients (tolerance 2 % of the reference's largest value,
the bf16 rounding of the outputs), pool / upsample and their gradients,
the whole network's loss and weight gradients, and a short training run."""
import ctypes
import threading

import numpy as np
import pytest

import roxy_native as nat

torch = pytest.importorskip("torch")
F = torch.nn.functional
pytestmark = pytest.mark.gpu


def _ctx():
    return nat.context()


def _p(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


def _stream():
    # torch's default stream (handle 0) is the legacy default stream, handle 1
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream or 1)


def _close(got, ref, frac=2e-2):
    ref = ref.detach()
    scale = float(ref.abs().max()) + 1e-6
    err = float((got.float() - ref.float()).abs().max())
    assert err <= frac * scale, (err, scale)


def _view(t, off, c):
    return t[..., off:off + c]


CASES = [  # N, H, W, Cin, Cout, x_stride, x_off, y_stride, y_off, relu
    (1, 8, 8, 16, 32, 16, 0, 32, 0, 1),
    (2, 17, 23, 32, 64, 48, 16, 64, 0, 0),
    (1, 12, 20, 64, 128, 64, 0, 160, 32, 1),
    (1, 9, 31, 192, 64, 192, 0, 96, 32, 1),
    (2, 16, 16, 96, 16, 96, 0, 16, 0, 0),
    (1, 40, 36, 128, 128, 128, 0, 128, 0, 1),
]


@pytest.fixture(params=[0, 1, 2], ids=["tcgen05", "mma_sync", "tcgen05_streaming"])
def impl(request):
    ctx = _ctx()
    ctx.check(nat.lib().rx_conv_set_impl(ctx.h, request.param))
    yield request.param
    ctx.check(nat.lib().rx_ctx_sync(ctx.h))  # no kernel raised its error flag
    ctx.check(nat.lib().rx_conv_set_impl(ctx.h, 0))


@pytest.mark.parametrize("N,H,W,Cin,Cout,xs,xo,ys,yo,relu", CASES + [(1, 3, 300, 32, 64, 32, 0, 64, 0, 1)])
def test_conv_fwd_and_grads_match_torch(N, H, W, Cin, Cout, xs, xo, ys, yo, relu, impl):
    ctx = _ctx()
    g = torch.Generator(device="cuda").manual_seed(N * 1000 + H)
    dev = "cuda"
    xbuf = torch.randn((N, H, W, xs), generator=g, device=dev).to(torch.bfloat16)
    w = (torch.randn((Cout, 9, Cin), generator=g, device=dev) * (1.0 / np.sqrt(9 * Cin))).to(torch.bfloat16)
    bias = torch.randn(Cout, generator=g, device=dev) * 0.1
    ybuf = torch.zeros((N, H, W, ys), dtype=torch.bfloat16, device=dev)
    d = nat.ConvDesc(N, H, W, Cin, Cout, xs, xo, ys, yo)
    L = nat.lib()
    ctx.check(L.rx_conv_bf16_fwd(ctx.h, ctypes.byref(d), _p(xbuf), _p(w), _p(bias), _p(ybuf), None, relu, _stream()))
    xin = _view(xbuf, xo, Cin).float().permute(0, 3, 1, 2).contiguous().requires_grad_(True)
    wt = w.float().view(Cout, 3, 3, Cin).permute(0, 3, 1, 2).contiguous().requires_grad_(True)
    bt = bias.clone().requires_grad_(True)
    ref = F.conv2d(xin, wt, bt, padding=1)
    if relu:
        ref = F.relu(ref)
    got = _view(ybuf, yo, Cout).float().permute(0, 3, 1, 2)
    torch.cuda.synchronize()
    _close(got, ref)
    # untouched channels of the output view stay zero
    if ys > Cout:
        mask = torch.ones(ys, dtype=torch.bool, device=dev)
        mask[yo:yo + Cout] = False
        assert float(ybuf[..., mask].float().abs().max()) == 0.0
    # gradients for a random output gradient
    dyv = torch.randn((N, H, W, Cout), generator=g, device=dev).to(torch.bfloat16)
    dybuf = torch.zeros((N, H, W, ys), dtype=torch.bfloat16, device=dev)
    dybuf[..., yo:yo + Cout] = dyv
    ref.backward(dyv.float().permute(0, 3, 1, 2))
    dxbuf = torch.zeros((N, H, W, xs), dtype=torch.bfloat16, device=dev)
    rot = torch.empty(Cout * 9 * Cin, dtype=torch.bfloat16, device=dev)
    dw = torch.zeros((Cout, 9, Cin), dtype=torch.float32, device=dev)
    db = torch.zeros(Cout, dtype=torch.float32, device=dev)
    if relu:
        # the kernels take the gradient after the ReLU mask
        op = nat.DnOp(nat.RX_DN_RELU_MASK, N, H, W, Cout, _p(ybuf), ys, yo, _p(dybuf), ys, yo, 0)
        ctx.check(L.rx_dn_layer(ctx.h, ctypes.byref(op), _stream()))
    ctx.check(L.rx_conv_bf16_bwd_data(ctx.h, ctypes.byref(d), _p(dybuf), _p(w), _p(rot), _p(dxbuf), _stream()))
    ctx.check(L.rx_conv_bf16_bwd_weight(ctx.h, ctypes.byref(d), _p(dybuf), _p(xbuf), _p(dw), _p(db), _stream()))
    torch.cuda.synchronize()
    _close(_view(dxbuf, xo, Cin).float().permute(0, 3, 1, 2), xin.grad, 3e-2)
    _close(dw.view(Cout, 3, 3, Cin).permute(0, 3, 1, 2), wt.grad, 2e-2)
    _close(db, bt.grad, 2e-2)


def test_conv_rejects_bad_descriptors():
    ctx = _ctx()
    x = torch.zeros((1, 4, 4, 16), dtype=torch.bfloat16, device="cuda")
    w = torch.zeros((16, 9, 16), dtype=torch.bfloat16, device="cuda")
    for d in (nat.ConvDesc(1, 4, 4, 12, 16, 16, 0, 16, 0), nat.ConvDesc(1, 4, 4, 16, 16, 16, 4, 16, 0),
              nat.ConvDesc(1, 4, 4, 16, 16, 16, 0, 8, 0)):
        with pytest.raises(ValueError):
            ctx.check(nat.lib().rx_conv_bf16_fwd(ctx.h, ctypes.byref(d), _p(x), _p(w), None, _p(x), None, 0, None))


def test_pool_and_upsample_match_torch():
    ctx = _ctx()
    L = nat.lib()
    N, H, W, C = 2, 12, 20, 32
    x = torch.randn((N, H, W, C), device="cuda").to(torch.bfloat16)
    p = torch.zeros((N, H // 2, W // 2, C), dtype=torch.bfloat16, device="cuda")
    ctx.check(L.rx_dn_layer(ctx.h, ctypes.byref(nat.DnOp(nat.RX_DN_POOL, N, H, W, C, _p(x), C, 0, _p(p), C, 0, 0)),
                            _stream()))
    u = torch.zeros((N, 2 * H, 2 * W, C), dtype=torch.bfloat16, device="cuda")
    ctx.check(L.rx_dn_layer(ctx.h, ctypes.byref(nat.DnOp(nat.RX_DN_UP, N, H, W, C, _p(x), C, 0, _p(u), C, 0, 0)),
                            _stream()))
    xt = x.float().permute(0, 3, 1, 2)
    _close(p.float().permute(0, 3, 1, 2), F.avg_pool2d(xt, 2), 1e-2)
    _close(u.float().permute(0, 3, 1, 2), F.interpolate(xt, scale_factor=2, mode="nearest"), 1e-6)
    # channel views (16-byte chunk kernels) and a stride that is not a
    # multiple of 8 channels (element kernels): the same values
    for stride, off in ((48, 16), (36, 4)):
        wide = torch.zeros((N, H, W, stride), dtype=torch.bfloat16, device="cuda")
        wide[..., off:off + C] = x
        pv = torch.zeros((N, H // 2, W // 2, stride), dtype=torch.bfloat16, device="cuda")
        uv = torch.zeros((N, 2 * H, 2 * W, stride), dtype=torch.bfloat16, device="cuda")
        ctx.check(L.rx_dn_layer(ctx.h, ctypes.byref(nat.DnOp(nat.RX_DN_POOL, N, H, W, C, _p(wide), stride, off,
                                                             _p(pv), stride, off, 0)), _stream()))
        ctx.check(L.rx_dn_layer(ctx.h, ctypes.byref(nat.DnOp(nat.RX_DN_UP, N, H, W, C, _p(wide), stride, off,
                                                             _p(uv), stride, off, 0)), _stream()))
        torch.cuda.synchronize()
        assert torch.equal(pv[..., off:off + C], p) and torch.equal(uv[..., off:off + C], u), (stride, off)
        assert not pv[..., :off].any() and not uv[..., off + C:].any()
    # gradients
    gp = torch.randn((N, H // 2, W // 2, C), device="cuda").to(torch.bfloat16)
    gx = torch.zeros_like(x)
    ctx.check(L.rx_dn_layer(ctx.h, ctypes.byref(nat.DnOp(nat.RX_DN_POOL_BWD, N, H, W, C, _p(gp), C, 0, _p(gx), C, 0,
                                                         0)), _stream()))
    xr = xt.clone().requires_grad_(True)
    F.avg_pool2d(xr, 2).backward(gp.float().permute(0, 3, 1, 2))
    _close(gx.float().permute(0, 3, 1, 2), xr.grad, 1e-2)
    gu = torch.randn((N, 2 * H, 2 * W, C), device="cuda").to(torch.bfloat16)
    gx2 = torch.zeros_like(x)
    ctx.check(L.rx_dn_layer(ctx.h, ctypes.byref(nat.DnOp(nat.RX_DN_UP_BWD, N, H, W, C, _p(gu), C, 0, _p(gx2), C, 0,
                                                         0)), _stream()))
    xr2 = xt.clone().requires_grad_(True)
    F.interpolate(xr2, scale_factor=2, mode="nearest").backward(gu.float().permute(0, 3, 1, 2))
    torch.cuda.synchronize()
    _close(gx2.float().permute(0, 3, 1, 2), xr2.grad, 1e-2)


def _torch_net(net, x16, base, target):
    """fp32 PyTorch replica of the network on the same bf16 weights."""
    from rendering.learned_denoiser import LAYERS
    params = {}
    for name, cin, cout, _ in LAYERS:
        w = net.w16[name].float().view(cout, 3, 3, cin).permute(0, 3, 1, 2).contiguous().requires_grad_(True)
        b = net.b32[name].clone().requires_grad_(True)
        params[name] = (w, b)

    def conv(name, t, relu=True):
        w, b = params[name]
        y = F.conv2d(t, w, b, padding=1)
        return F.relu(y) if relu else y

    x = x16.float().permute(0, 3, 1, 2)
    s1 = conv("e1b", conv("e1a", x))
    s2 = conv("e2b", conv("e2a", F.avg_pool2d(s1, 2)))
    e3 = conv("e3b", conv("e3a", F.avg_pool2d(s2, 2)))
    d2 = conv("d2b", conv("d2a", torch.cat([F.interpolate(e3, scale_factor=2), s2], 1)))
    d1 = conv("d1b", conv("d1a", torch.cat([F.interpolate(d2, scale_factor=2), s1], 1)))
    out = conv("head", d1, relu=False)[:, :3].permute(0, 2, 3, 1)
    loss = (out + base - target).abs().sum()
    P = x.shape[0] * x.shape[2] * x.shape[3]
    (loss / (3 * P)).backward()
    return float(loss.detach()), {k: (v[0].grad, v[1].grad) for k, v in params.items()}


@pytest.mark.parametrize("N,H,W,C,stride,off", [(1, 2, 2, 8, 8, 0), (2, 6, 10, 24, 48, 16), (3, 2, 34, 32, 40, 8),
                                                (1, 66, 130, 128, 192, 64)])
def test_chunked_layer_gradients_equal_the_element_kernels(N, H, W, C, stride, off):
    """ReLU mask, pool and upsample gradients on 8-channel chunks give the
    bits of the element kernels (reached by a stride that is no multiple of
    8) and leave the other channels alone."""
    ctx, L = _ctx(), nat.lib()
    g = torch.Generator(device="cuda").manual_seed(N * 100 + C)
    rnd = lambda *s: torch.randn(s, device="cuda", generator=g).to(torch.bfloat16)  # noqa: E731
    y, big, small = rnd(N, H, W, C), rnd(N, H, W, C), rnd(N, H // 2, W // 2, C)
    y.view(-1)[::7] = 0.0
    y.view(-1)[3::11] = float("nan")

    def run(kind, n, h, w, a, b, flag, st, of):
        wide = lambda t: F.pad(t, (of, st - of - C), value=3.0).contiguous()  # noqa: E731
        aw, bw = wide(a), wide(b)
        ctx.check(L.rx_dn_layer(ctx.h, ctypes.byref(nat.DnOp(kind, n, h, w, C, _p(aw), st, of, _p(bw), st, of, flag)),
                                _stream()))
        torch.cuda.synchronize()
        assert bool((bw[..., :of] == 3.0).all()) and bool((bw[..., of + C:] == 3.0).all())
        return bw[..., of:of + C].contiguous().view(torch.int16)

    for kind, n, h, w, a, b, flag in ((nat.RX_DN_RELU_MASK, N, H, W, y, big, 0),
                                      (nat.RX_DN_POOL_BWD, N, H, W, small, big, 0),
                                      (nat.RX_DN_POOL_BWD, N, H, W, small, big, 1),
                                      (nat.RX_DN_UP_BWD, N, H // 2, W // 2, big, small, 0)):
        assert torch.equal(run(kind, n, h, w, a, b, flag, stride, off),
                           run(kind, n, h, w, a, b, flag, stride + 4, off + 2)), kind


@pytest.mark.parametrize("P", [1, 4, 6, 1028])
def test_features_and_loss_chunks_equal_the_element_kernels(P):
    """Four pixels per item (P a multiple of 4, aligned planes) against the
    same pixels one by one (planes shifted by one pixel), and the loss
    gradient in 16-byte stores against stride 12."""
    ctx, L = _ctx(), nat.lib()
    g = torch.Generator(device="cuda").manual_seed(P)
    planes = [torch.rand((P + 1, k), device="cuda", generator=g) * 4 - 1 for k in (3, 3, 3, 1)]

    def feats(ts):
        out, base = (torch.empty((P, k), dtype=d, device="cuda") for k, d in ((16, torch.bfloat16), (3, torch.float32)))
        ctx.check(L.rx_dn_features(ctx.h, P, *[_p(t) for t in ts], _p(out), _p(base), _stream()))
        torch.cuda.synchronize()
        return out.view(torch.int16), base

    a, b = feats([t[1:].contiguous() for t in planes]), feats([t[1:] for t in planes])
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
    y32, t = torch.randn((P, 16), device="cuda", generator=g), torch.rand((P, 3), device="cuda", generator=g)
    grads = []
    for gs in (16, 12):
        gr = torch.full((P, gs), 5.0, dtype=torch.bfloat16, device="cuda")
        loss = torch.zeros(1, device="cuda")
        ctx.check(L.rx_dn_l1_loss(ctx.h, P, _p(y32), 16, _p(a[1]), _p(t), ctypes.c_float(0.5), _p(gr), gs, _p(loss),
                                  _stream()))
        torch.cuda.synchronize()
        assert not gr[:, 3:].any()
        grads.append(gr[:, :3].clone())
    assert torch.equal(*grads)


def test_tcgen05_and_mma_sync_convolutions_agree():
    """The forward kernels on the same operands (persistent and streaming
    tcgen05, then mma.sync): same values up to the order of their float32
    sums (and the bf16 rounding of the output)."""
    ctx = _ctx()
    L = nat.lib()
    g = torch.Generator(device="cuda").manual_seed(21)
    for (Cin, Cout, H, W) in ((16, 32, 33, 257), (96, 32, 20, 128), (64, 128, 9, 200), (32, 16, 5, 130),
                              (64, 64, 70, 300), (192, 64, 6, 129), (32, 32, 128, 512), (96, 32, 600, 256),
                              (96, 64, 20, 140), (128, 128, 12, 140)):
        x = torch.randn((2, H, W, Cin), generator=g, device="cuda").to(torch.bfloat16)
        w = (torch.randn((Cout, 9, Cin), generator=g, device="cuda") / np.sqrt(9 * Cin)).to(torch.bfloat16)
        b = torch.randn(Cout, generator=g, device="cuda")
        d = nat.ConvDesc(2, H, W, Cin, Cout, Cin, 0, Cout, 0)
        outs = []
        for impl_ in (0, 2, 1):
            ctx.check(L.rx_conv_set_impl(ctx.h, impl_))
            y = torch.zeros((2, H, W, Cout), dtype=torch.bfloat16, device="cuda")
            y32 = torch.zeros((2, H, W, Cout), dtype=torch.float32, device="cuda")
            ctx.check(L.rx_conv_bf16_fwd(ctx.h, ctypes.byref(d), _p(x), _p(w), _p(b), _p(y), _p(y32), 0, _stream()))
            outs.append(y32)
        ctx.check(L.rx_conv_set_impl(ctx.h, 0))
        ctx.check(L.rx_ctx_sync(ctx.h))
        scale = float(outs[2].abs().max())
        assert float((outs[0] - outs[2]).abs().max()) <= 1e-3 * scale, (Cin, Cout)
        assert float((outs[1] - outs[2]).abs().max()) <= 1e-3 * scale, (Cin, Cout)


def test_network_loss_and_gradients_match_torch():
    from rendering.learned_denoiser import LAYERS, Denoiser
    net = Denoiser(seed=3)
    N, H, W = 2, 16, 24
    g = torch.Generator(device="cuda").manual_seed(7)
    rad = torch.rand((N, H, W, 3), generator=g, device="cuda") * 2
    alb = torch.rand((N, H, W, 3), generator=g, device="cuda")
    nrm = torch.randn((N, H, W, 3), generator=g, device="cuda")
    dep = torch.rand((N, H, W, 1), generator=g, device="cuda") * 3
    target = torch.log1p(rad * 0.8 + 0.1)
    net.features(rad, alb, nrm, dep, N, H, W, train=True)
    b = net.forward(N, H, W, train=True)
    loss = float(net.loss(N, H, W, target))
    net.backward(N, H, W)
    torch.cuda.synchronize()
    ref_loss, grads = _torch_net(net, b["x"], b["base"], target)
    assert abs(loss - ref_loss) <= 2e-2 * abs(ref_loss)
    for name, cin, cout, _ in LAYERS:
        gw = net.dw[name].view(cout, 3, 3, cin).permute(0, 3, 1, 2).flatten()
        rw = grads[name][0].flatten()
        cos = float(torch.dot(gw, rw) / (gw.norm() * rw.norm() + 1e-20))
        assert cos > 0.98, (name, cos)
        cb = float(torch.dot(net.db[name], grads[name][1]) / (net.db[name].norm() * grads[name][1].norm() + 1e-20))
        assert cb > 0.98 or float(grads[name][1].norm()) < 1e-6, (name, cb)


def test_training_reduces_the_loss():
    from rendering.learned_denoiser import Denoiser
    net = Denoiser(seed=1)
    N, H, W = 4, 32, 32
    g = torch.Generator(device="cuda").manual_seed(11)
    clean = torch.rand((N, H, W, 3), generator=g, device="cuda")
    clean = F.avg_pool2d(clean.permute(0, 3, 1, 2), 5, 1, 2).permute(0, 2, 3, 1).contiguous()
    noisy = (clean * (1 + 0.6 * torch.randn((N, H, W, 3), generator=g, device="cuda"))).clamp_min(0)
    alb = torch.ones((N, H, W, 3), device="cuda") * 0.5
    nrm = torch.zeros((N, H, W, 3), device="cuda")
    dep = torch.ones((N, H, W, 1), device="cuda")
    target = torch.log1p(clean)
    losses = [float(net.train_step(noisy, alb, nrm, dep, target, lr=3e-3)) for _ in range(60)]
    assert np.mean(losses[-10:]) < 0.7 * np.mean(losses[:5]), (losses[:5], losses[-10:])
    out = net.denoise(noisy, alb, nrm, dep)
    assert out.shape == (N, H, W, 3) and bool(torch.isfinite(out).all())


@pytest.mark.parametrize("P,Cout,stride,off", [(1, 16, 16, 0), (37, 48, 64, 8), (5000, 32, 32, 0), (263, 2064, 2064, 0),
                                               (70001, 16, 96, 64)])
def test_bias_gradient_sums_every_pixel(P, Cout, stride, off):
    """db over block, lane and chunk remainders.  An fp32 sum of n terms in
    any order is off by at most (n - 1) 2^-24 sum |term| (n 2^-24 covers the
    second-order terms here)."""
    ctx = _ctx()
    g = torch.Generator(device="cuda").manual_seed(P)
    dy = torch.randn((1, 1, P, stride), generator=g, device="cuda").to(torch.bfloat16)
    x = torch.zeros((1, 1, P, 16), dtype=torch.bfloat16, device="cuda")
    dw = torch.zeros((Cout, 9, 16), device="cuda")
    db = torch.ones(Cout, device="cuda")
    d = nat.ConvDesc(1, 1, P, 16, Cout, 16, 0, stride, off)
    ctx.check(nat.lib().rx_conv_bf16_bwd_weight(ctx.h, ctypes.byref(d), _p(dy), _p(x), _p(dw), _p(db), _stream()))
    torch.cuda.synchronize()
    v = _view(dy, off, Cout).double().reshape(P, Cout)
    bound = (P + 1) * 2.0 ** -24 * (v.abs().sum(0) + 1.0)
    assert bool(((db.double() - (v.sum(0) + 1.0)).abs() <= bound).all())


@pytest.mark.parametrize("N,H,W,Cin,Cout,xs,xo,ys,yo,y32", [
    (1, 1, 1, 16, 48, 16, 0, 48, 0, 1),        # one pixel; a group partly out of range
    (2, 3, 8, 32, 96, 40, 8, 104, 8, 0),       # narrow images: 16 rows of 8 pixels
    (3, 17, 33, 64, 192, 64, 0, 192, 0, 1),    # two groups of 96, ragged tiles
    (1, 5, 129, 32, 160, 32, 0, 160, 0, 0),    # one pixel beyond a tile
    (2, 128, 128, 32, 96, 32, 0, 96, 0, 0),    # more tiles than blocks
    (1, 40, 70, 16, 224, 16, 0, 224, 0, 0),    # groups of 64 and of 96 tie
])
def test_resident_weight_conv_tile_edges(N, H, W, Cin, Cout, xs, xo, ys, yo, y32):
    """The kernel that keeps a group's weights in shared memory, at its tiles'
    and groups' edges: bounds as for the warp-specialised kernel below."""
    test_warp_specialised_conv_tile_edges(N, H, W, Cin, Cout, xs, xo, ys, yo, y32)


@pytest.mark.parametrize("N,H,W,Cin,Cout,xs,xo,ys,yo,y32", [
    (1, 1, 1, 16, 16, 16, 0, 16, 0, 1),        # one pixel, one row
    (3, 2, 127, 32, 32, 40, 8, 40, 8, 0),      # one short tile; views off the 32-byte grid
    (2, 5, 128, 48, 64, 48, 0, 64, 0, 1),      # a whole tile; a step count outside the unrolled ones
    (1, 700, 129, 16, 32, 16, 0, 32, 0, 0),    # a second tile of one pixel, strips over several blocks
    (2, 3, 257, 96, 32, 112, 16, 96, 64, 0),   # six steps per tap
    (1, 33, 130, 64, 128, 64, 0, 128, 0, 0),   # the widest group
    (1, 7, 140, 192, 64, 192, 0, 64, 0, 1),    # split over the input channels
    (1, 4, 300, 160, 16, 160, 0, 16, 0, 0),    # many steps, narrow output
])
def test_warp_specialised_conv_tile_edges(N, H, W, Cin, Cout, xs, xo, ys, yo, y32):
    """Row strips, tiles and ring phases at their edges against float64.  The
    sum is fp32 over K = 9 Cin products (each add may truncate: K 2^-22 of
    the absolute sum), the bf16 output rounds by 2^-8 of the value."""
    ctx = _ctx()
    g = torch.Generator(device="cuda").manual_seed(H * 1000 + W)
    xbuf = torch.randn((N, H, W, xs), generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn((Cout, 9, Cin), generator=g, device="cuda") / np.sqrt(9 * Cin)).to(torch.bfloat16)
    bias = torch.randn(Cout, generator=g, device="cuda")
    ybuf = torch.zeros((N, H, W, ys), dtype=torch.bfloat16, device="cuda")
    f32 = torch.zeros((N, H, W, ys), device="cuda") if y32 else None
    d = nat.ConvDesc(N, H, W, Cin, Cout, xs, xo, ys, yo)
    ctx.check(nat.lib().rx_conv_bf16_fwd(ctx.h, ctypes.byref(d), _p(xbuf), _p(w), _p(bias), _p(ybuf), _p(f32), 0,
                                         _stream()))
    ctx.check(nat.lib().rx_ctx_sync(ctx.h))
    x = _view(xbuf, xo, Cin).double().permute(0, 3, 1, 2)
    wt = w.double().view(Cout, 3, 3, Cin).permute(0, 3, 1, 2)
    ref = F.conv2d(x, wt, bias.double(), padding=1).permute(0, 2, 3, 1)
    mag = F.conv2d(x.abs(), wt.abs(), bias.double().abs(), padding=1).permute(0, 2, 3, 1)
    tol = 9 * Cin * 2.0 ** -22 * mag
    got = _view(ybuf, yo, Cout).double()
    assert bool(((got - ref).abs() <= tol + 2.0 ** -8 * ref.abs()).all())
    if y32:
        assert bool(((_view(f32, yo, Cout).double() - ref).abs() <= tol).all())
    mask = torch.ones(ys, dtype=torch.bool, device="cuda")
    mask[yo:yo + Cout] = False
    assert not bool(ybuf[..., mask].any())


@pytest.mark.parametrize("N,H,W,Cin,Cout,xs,xo,ys,yo", [
    (1, 1, 1, 16, 16, 16, 0, 16, 0),          # one pixel: every tap but the centre reads zeros
    (2, 3, 17, 32, 32, 40, 8, 48, 16),        # a 32-pixel tile with 15 of them past the image
    (1, 2, 129, 96, 32, 96, 0, 32, 0),        # a second tile of one pixel
    (3, 90, 130, 16, 48, 16, 0, 48, 0),       # strips over several blocks and images, three output groups
    (1, 5, 300, 64, 64, 64, 0, 64, 0),        # nine taps in two groups
    (2, 9, 33, 128, 128, 128, 0, 192, 64),    # nine taps in three groups, four x slots
    (1, 6, 40, 272, 96, 272, 0, 96, 0),       # three input groups, the last one short
    (1, 4, 20, 144, 256, 144, 0, 256, 0),     # two input and two output groups
])
def test_weight_gradient_tile_edges(N, H, W, Cin, Cout, xs, xo, ys, yo):
    """dw += the float64 gradient, over tiles, strips and channel groups.  An
    fp32 sum of N H W products whose adds may truncate is off by at most
    2^-22 N H W of the absolute sum."""
    ctx = _ctx()
    g = torch.Generator(device="cuda").manual_seed(H * 1000 + W)
    x = torch.randn((N, H, W, xs), generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randn((N, H, W, ys), generator=g, device="cuda").to(torch.bfloat16)
    dw = torch.ones((Cout, 9, Cin), device="cuda")
    d = nat.ConvDesc(N, H, W, Cin, Cout, xs, xo, ys, yo)
    ctx.check(nat.lib().rx_conv_bf16_bwd_weight(ctx.h, ctypes.byref(d), _p(dy), _p(x), _p(dw), None, _stream()))
    ctx.check(nat.lib().rx_ctx_sync(ctx.h))
    xv = F.pad(_view(x, xo, Cin).double(), (0, 0, 1, 1, 1, 1))
    dv = _view(dy, yo, Cout).double().reshape(-1, Cout)
    for tap in range(9):
        cols = xv[:, tap // 3:tap // 3 + H, tap % 3:tap % 3 + W].reshape(-1, Cin)
        ref, mag = dv.t() @ cols, dv.abs().t() @ cols.abs()
        assert bool(((dw[:, tap].double() - 1.0 - ref).abs() <= (N * H * W + 2) * 2.0 ** -22 * (mag + 1.0)).all()), tap


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("N,H,W,Cin,Cout,xs,xo", [
    (1, 3, 1, 16, 16, 16, 0),       # one column: no product of the left taps at all
    (1, 4, 17, 32, 32, 48, 16),     # a whole step and one pixel
    (2, 3, 40, 96, 64, 96, 0),      # half a last step
    (1, 3, 125, 128, 128, 128, 0),  # eight steps, the last one short
    (1, 2, 130, 48, 16, 48, 0),     # the second tile's last step
    (1, 3, 48, 64, 48, 64, 0),      # no short step
])
def test_weight_gradient_takes_only_products_of_the_image(N, H, W, Cin, Cout, xs, xo, bad):
    """A non-finite activation in the last column enters the gradient of the
    taps that read it for some output pixel and of no other: the left taps
    (tap column 0) read the column to the left of a pixel, so never the
    last.  Their gradient is that of the activations without it."""
    ctx = _ctx()
    g = torch.Generator(device="cuda").manual_seed(W)
    x = torch.randint(-3, 4, (N, H, W, xs), generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randint(-3, 4, (N, H, W, Cout), generator=g, device="cuda").to(torch.bfloat16)
    dws = []
    for v in (0.0, bad):
        x[:, :, W - 1, xo:xo + Cin:3] = v
        dw = torch.zeros((Cout, 9, Cin), device="cuda")
        d = nat.ConvDesc(N, H, W, Cin, Cout, xs, xo, Cout, 0)
        ctx.check(nat.lib().rx_conv_bf16_bwd_weight(ctx.h, ctypes.byref(d), _p(dy), _p(x), _p(dw), None, _stream()))
        ctx.check(nat.lib().rx_ctx_sync(ctx.h))
        dws.append(dw)
    for tap in (0, 3, 6):
        assert torch.equal(dws[0][:, tap], dws[1][:, tap]), tap
    for tap in (1, 4, 7):
        hit = torch.isfinite(dws[1][:, tap]).logical_not()
        assert not hit[:, 1::3].any() and hit[:, 0::3].any()


def test_resident_weight_conv_from_several_threads():
    """Eight threads, each with its own context and stream, on two sizes whose
    tiles ask for different amounts of shared memory: every call is accepted
    and gives the bits it gives alone."""
    cases = [(1, 128, 128, 64, 192), (1, 16, 8, 64, 192)] * 4
    g = torch.Generator(device="cuda").manual_seed(5)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    data = [(rnd(n, h, w, ci), rnd(co, 9, ci), torch.empty((n, h, w, co), dtype=torch.bfloat16, device="cuda"))
            for n, h, w, ci, co in cases]
    ctxs = [nat.Context(0) for _ in cases]
    fails, want = [0] * len(cases), []

    def work(i, times):
        n, h, w, ci, co = cases[i]
        d = nat.ConvDesc(n, h, w, ci, co, ci, 0, co, 0)
        x, wt, y = data[i]
        args = (ctxs[i].h, ctypes.byref(d), _p(x), _p(wt), None, _p(y), None, 0, ctypes.c_void_p(ctxs[i].stream))
        for _ in range(times):
            fails[i] += nat.lib().rx_conv_bf16_fwd(*args) != 0

    torch.cuda.synchronize()
    for i in range(len(cases)):
        work(i, 1)
        ctxs[i].sync()
        want.append(data[i][2].clone())
        data[i][2].zero_()
    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(i, 4000)) for i in range(len(cases))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for c in ctxs:
        c.sync()
    assert not any(fails)
    assert all(torch.equal(data[i][2], want[i]) for i in range(len(cases)))


def test_unaligned_buffers_are_refused_or_served(impl):
    """What the kernels copy in 16-byte pieces is refused where it does not
    start on such a boundary, before anything is enqueued; an output on a
    4-byte one is served, with the bits of an aligned one."""
    ctx, L = _ctx(), nat.lib()
    N, H, W, ci, co = 1, 5, 33, 64, 32
    g = torch.Generator(device="cuda").manual_seed(8)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    x, w, dy = rnd(N * H * W * ci + 8), rnd(co * 9 * ci + 8), rnd(N * H * W * co + 8)
    rot, y = torch.zeros_like(w), torch.zeros_like(dy)
    dw, db, bias = torch.zeros((co, 9, ci), device="cuda"), torch.zeros(co, device="cuda"), torch.zeros(co, device="cuda")
    at = lambda t, n: ctypes.c_void_p(t.data_ptr() + n)  # noqa: E731
    d = ctypes.byref(nat.ConvDesc(N, H, W, ci, co, ci, 0, co, 0))
    fwd = lambda a, b, c: L.rx_conv_bf16_fwd(ctx.h, d, at(x, a), at(w, b), _p(bias), at(y, c), None, 0, _stream())  # noqa: E731
    bwd = lambda a, b, c: L.rx_conv_bf16_bwd_data(ctx.h, d, at(dy, a), at(w, 2), at(rot, b), at(x, c), _stream())  # noqa: E731
    wgt = lambda a, b: L.rx_conv_bf16_bwd_weight(ctx.h, d, at(dy, a), at(x, b), _p(dw), _p(db), _stream())  # noqa: E731
    keep = x.clone()
    for k in (2, 4, 8):
        assert fwd(k, 0, 0) == fwd(0, k, 0) == bwd(k, 0, 0) == bwd(0, k, 0) == wgt(k, 0) == wgt(0, k) == nat.RX_ERR_ARG
    assert fwd(0, 0, 2) == bwd(0, 0, 2) == nat.RX_ERR_ARG
    torch.cuda.synchronize()
    assert not rot.any() and not y.any() and not dw.any() and torch.equal(x, keep)
    assert fwd(0, 0, 4) == 0
    torch.cuda.synchronize()
    off = y[2:2 + N * H * W * co].clone()
    ctx.check(L.rx_conv_set_impl(ctx.h, 1))
    assert fwd(0, 0, 0) == 0
    torch.cuda.synchronize()
    assert torch.equal(off, y[:N * H * W * co]) and bool(off.any())
    assert bwd(0, 0, 4) == 0 and wgt(0, 0) == 0
    ctx.sync()


@pytest.mark.parametrize("P,Cout,stride,off", [(1, 16, 16, 0), (37, 48, 64, 8), (70001, 16, 96, 64), (263, 2064, 2064, 0),
                                               (262147, 16, 16, 0), (100003, 48, 48, 0)])
def test_bias_gradient_is_exact_on_small_integers(P, Cout, stride, off):
    """Sums of integers below 2^24 are exact in any order, so a pixel that is
    lost or taken twice -- in a lane, block or cluster, eight of those from
    229,377 pixels of 16 channels on -- shows."""
    ctx = _ctx()
    g = torch.Generator(device="cuda").manual_seed(P)
    dy = torch.randint(1, 4, (1, 1, P, stride), generator=g, device="cuda").to(torch.bfloat16)
    x = torch.zeros((1, 1, P, 16), dtype=torch.bfloat16, device="cuda")
    dw, db = torch.zeros((Cout, 9, 16), device="cuda"), torch.ones(Cout, device="cuda")
    d = nat.ConvDesc(1, 1, P, 16, Cout, 16, 0, stride, off)
    ctx.check(nat.lib().rx_conv_bf16_bwd_weight(ctx.h, ctypes.byref(d), _p(dy), _p(x), _p(dw), _p(db), _stream()))
    ctx.check(nat.lib().rx_ctx_sync(ctx.h))
    assert torch.equal(db.double(), _view(dy, off, Cout).double().reshape(P, Cout).sum(0) + 1.0)


@pytest.mark.parametrize("N,H,W,Cin,Cout,xs,xo,ys,yo", [
    (3, 90, 130, 16, 48, 16, 0, 48, 0),       # strips over several blocks and images, a two-pixel second tile
    (2, 100, 128, 96, 32, 96, 0, 32, 0),      # whole tiles
    (5, 64, 64, 64, 64, 72, 8, 96, 32),       # several taps' groups
    (2, 57, 33, 128, 128, 128, 0, 192, 64),
    (1, 61, 300, 272, 16, 272, 0, 16, 0),     # three input groups
])
def test_weight_gradient_is_exact_on_small_integers(N, H, W, Cin, Cout, xs, xo, ys, yo):
    """The same for the weight gradient: products of integers up to 3, sums
    below 2^24, so a row, a strip's end or an image border that is lost,
    taken twice or shifted shows."""
    assert 9 * N * H * W < 2 ** 24
    ctx = _ctx()
    g = torch.Generator(device="cuda").manual_seed(H * 1000 + W)
    x = torch.randint(-3, 4, (N, H, W, xs), generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randint(-3, 4, (N, H, W, ys), generator=g, device="cuda").to(torch.bfloat16)
    dw = torch.ones((Cout, 9, Cin), device="cuda")
    d = nat.ConvDesc(N, H, W, Cin, Cout, xs, xo, ys, yo)
    ctx.check(nat.lib().rx_conv_bf16_bwd_weight(ctx.h, ctypes.byref(d), _p(dy), _p(x), _p(dw), None, _stream()))
    ctx.check(nat.lib().rx_ctx_sync(ctx.h))
    xv = F.pad(_view(x, xo, Cin).double(), (0, 0, 1, 1, 1, 1))
    dv = _view(dy, yo, Cout).double().reshape(-1, Cout)
    for tap in range(9):
        cols = xv[:, tap // 3:tap // 3 + H, tap % 3:tap % 3 + W].reshape(-1, Cin)
        assert torch.equal(dw[:, tap].double(), dv.t() @ cols + 1.0), tap


@pytest.mark.parametrize("P", [1, 1023, 1025, 151_553, 262_147])
@pytest.mark.parametrize("gs,with_base", [(16, True), (12, False)])
def test_loss_is_exact_on_quarters(P, gs, with_base):
    """Distances that are multiples of 1/4 with a sum below 2^22: exact in
    float32, so a pixel or block that the reduction loses shows; up to more
    pixels than one per thread of a block per SM."""
    ctx = _ctx()
    g = torch.Generator(device="cuda").manual_seed(P)
    quarters = lambda *s: torch.randint(-4, 5, s, generator=g, device="cuda").float() / 4  # noqa: E731
    y32, base, t = quarters(P, 16), quarters(P, 3) if with_base else None, quarters(P, 3)
    gr = torch.empty((P, gs), dtype=torch.bfloat16, device="cuda")
    loss = torch.ones(1, device="cuda")
    ctx.check(nat.lib().rx_dn_l1_loss(ctx.h, P, _p(y32), 16, _p(base), _p(t), ctypes.c_float(0.5), _p(gr), gs,
                                      _p(loss), _stream()))
    torch.cuda.synchronize()
    dlt = y32[:, :3].double() + (base.double() if with_base else 0.0) - t.double()
    want = dlt.abs().sum() + 1.0
    assert want < 2 ** 22 and float(loss) == float(want)
    assert torch.equal(gr[:, :3].double(), torch.sign(dlt) * 0.5)
