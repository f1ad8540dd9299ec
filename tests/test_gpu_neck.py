"""GPU: the kernels between the dense convolutions of the 2D neck, at the edges of their tiles, against torch in fp32.

Layout and bias + ReLU (+ sum) round where separate fp16 operations round: bit for bit. The attention and the heads sum 128
products in fp32, in another order than torch (128 * 2^-24 of the sum of magnitudes), and then round to fp16 (2^-11 of the
value) after the sum, after the bias, the attention's weights, its two products and their sum."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,channels,pixels", [(1, 8, 1), (2, 64, 63), (1, 72, 65), (3, 128, 129), (1, 128, 202 * 178)])
def test_channels_last(gpu, batch, channels, pixels):
    import torch

    x = torch.randn((batch, channels, pixels), device="cuda").half()
    y = torch.empty((batch, pixels, channels), device="cuda", dtype=torch.float16)
    assert gpu.lib().sessd_channels_last_enqueue(x.data_ptr(), y.data_ptr(), batch, channels, pixels, gpu._stream()) == 0
    assert torch.equal(y, x.transpose(1, 2))


@pytest.mark.parametrize("add", [False, True])
@pytest.mark.parametrize("pixels,channels", [(1, 8), (33, 128), (100 * 88, 256), (200 * 176 * 3 + 1, 128)])
def test_bias_relu(gpu, pixels, channels, add):
    import torch

    y = torch.randn((pixels, channels), device="cuda").half()
    bias = torch.randn(channels, device="cuda").half()
    other = torch.randn((pixels, channels), device="cuda").half() if add else None
    want = torch.relu(y + bias)
    want = want + other if add else want
    assert gpu.lib().sessd_bias_relu_enqueue(y.data_ptr(), bias.data_ptr(), other.data_ptr() if add else None, pixels, channels,
                                             gpu._stream()) == 0
    assert torch.equal(y, want)
    assert gpu.lib().sessd_bias_relu_enqueue(y.data_ptr(), bias.data_ptr(), None, pixels, 24, gpu._stream()) != 0


def test_bias_relu_keeps_what_is_not_a_number(gpu):
    import torch

    inf, nan = float("inf"), float("nan")
    row = torch.tensor([nan, inf, -inf, 1.0, -1.0, 65504.0, -65504.0, 0.0], device="cuda").half()
    bias = torch.tensor([[0.0] * 8, [inf] * 8, [-inf] * 8, [nan] * 8, [65504.0] * 8], device="cuda").half()
    for b in bias:
        for add in (None, row.flip(0).expand(8, 8).contiguous()):
            y = row.expand(8, 8).contiguous()
            want = torch.relu(y + b)
            want = want if add is None else want + add
            assert gpu.lib().sessd_bias_relu_enqueue(y.data_ptr(), b.clone().data_ptr(), None if add is None else add.data_ptr(), 8, 8,
                                                     gpu._stream()) == 0
            assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y.nan_to_num(7.0), want.nan_to_num(7.0))


@pytest.mark.parametrize("pixels", [1, 63, 64, 65, 2 * 200 * 176 + 7])
def test_neck_tail(gpu, pixels):
    import torch

    g = torch.Generator(device="cuda").manual_seed(pixels)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").half()
    o0, o1, gw, gb, hw, hb = rnd(pixels, 128), rnd(pixels, 128), rnd(2, 128) * 0.1, rnd(2), rnd(22, 128) * 0.1, rnd(22)
    feat = torch.empty_like(o0)
    heads = [torch.empty((pixels, c), device="cuda") for c in (14, 2, 2, 4)]
    run = lambda f, h: gpu.lib().sessd_neck_tail_enqueue(gpu._vp(o0, o1, gw, gb, hw, hb), gpu._vp(f, *h), pixels, gpu._stream())
    assert run(feat, heads) == 0
    d = lambda t: t.double()
    logit = torch.stack([(d(o0) * d(gw[0])).sum(1) + d(gb[0]), (d(o1) * d(gw[1])).sum(1) + d(gb[1])], 1)
    w = torch.softmax(logit, 1)
    want = d(o0) * w[:, :1] + d(o1) * w[:, 1:]
    # a logit: its sum's error, two roundings; a weight moves by at most a quarter of the logits' errors, and is rounded
    mag = lambda o, w, b: (d(o).abs() @ d(w).abs().T + d(b).abs())
    slack = (128 * 2.0 ** -24 + 2 * 2.0 ** -11) * (mag(o0, gw[:1], gb[:1]) + mag(o1, gw[1:], gb[1:]))
    tol = (d(o0).abs() + d(o1).abs()) * (slack / 4 + 2.0 ** -11 + 2 * 2.0 ** -11) + 2.0 ** -23
    assert ((d(feat) - want).abs() <= tol).all()
    out = d(feat) @ d(hw).T + d(hb)
    tol = (129 * 2.0 ** -24 + 2 * 2.0 ** -11) * mag(feat, hw, hb) + 2.0 ** -23
    assert ((d(torch.cat(heads, 1)) - out).abs() <= tol).all()
    only = [torch.empty_like(h) for h in heads]
    assert run(None, only) == 0 and all(torch.equal(a, b) for a, b in zip(only, heads))
    only_feat = torch.empty_like(feat)
    assert run(only_feat, [None] * 4) == 0 and torch.equal(only_feat, feat)
    assert run(None, [None] * 4) != 0


@pytest.fixture(scope="module")
def neck(gpu):
    return gpu.detector.Neck2D(gpu.detector.random_neck_weights())


def _bev(batch, height, width, seed=3):
    import torch

    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn((batch, 128, height, width), generator=g, device="cuda").relu().half()


def test_heads_are_fp32_whatever_the_default_type(gpu, neck):
    import torch

    x = _bev(2, 18, 26)
    want = neck(x)
    try:
        torch.set_default_dtype(torch.float64)
        got = neck(x)
    finally:
        torch.set_default_dtype(torch.float32)
    for k, v in want.items():
        assert v.dtype == got[k].dtype == torch.float32 and torch.equal(v, got[k])


def test_weights_written_just_before_the_call(gpu):
    """Bias and weights that the kernel launched just before writes (its blocks let the next kernel start early)."""
    import torch

    lib, s = gpu.lib(), gpu._stream()
    zero = torch.zeros(128, dtype=torch.float16, device="cuda")
    big = torch.zeros((300000, 128), dtype=torch.float16, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(1)
    o0, o1 = (torch.randn((64, 128), generator=g, device="cuda").half() for _ in range(2))
    for i in range(1, 20):
        params = torch.full((26, 128), i / 64.0, dtype=torch.float16, device="cuda")     # 2 gate rows, gate and head bias, 22 head rows
        big.zero_()
        big[-26:].fill_(-1.0)
        y = torch.zeros((64, 128), dtype=torch.float16, device="cuda")
        heads = [torch.empty((64, c), device="cuda") for c in (14, 2, 2, 4)]
        want = [torch.empty_like(h) for h in heads]
        run = lambda w, out: lib.sessd_neck_tail_enqueue(gpu._vp(o0, o1, w[:2], w[2], w[4:], w[3]), gpu._vp(None, *out), 64, s)
        assert run(params, want) == 0
        tail = big[-26:]
        add = torch.zeros_like(big)
        add[-26:] = params
        torch.cuda.synchronize()
        assert lib.sessd_bias_relu_enqueue(big.data_ptr(), zero.data_ptr(), add.data_ptr(), len(big), 128, s) == 0
        assert lib.sessd_bias_relu_enqueue(y.data_ptr(), tail[5].data_ptr(), None, 64, 128, s) == 0
        assert (y == i / 64.0).all()
        tail.fill_(-1.0)
        assert lib.sessd_bias_relu_enqueue(big.data_ptr(), zero.data_ptr(), add.data_ptr(), len(big), 128, s) == 0
        assert run(tail, heads) == 0
        assert all(torch.equal(a, b) for a, b in zip(heads, want))


def _close(got, want, tol=2.0 ** -8):
    """Kernels and separate operations round to fp16 at the same points; the attention's and the heads' sums may fall on the other
    side of a rounding (2^-11 of a weight, of its products, of a head's sum): a few of those."""
    assert got.dtype == want.dtype and got.shape == want.shape
    assert float((got - want).abs().max()) <= tol * float(want.abs().max())


def test_inputs_that_the_kernels_do_not_take(gpu, neck):
    """Gradients, forward mode, autocast, function transforms, an empty batch, the CPU, another type: as torch's operations do."""
    import torch

    D = gpu.detector
    x = _bev(2, 10, 14)
    want, heads = neck.features(x), neck(x)
    leaf = x.clone().requires_grad_()
    got = neck.features(leaf)
    _close(got.detach(), want)
    for k, v in neck(leaf).items():
        _close(v.detach(), heads[k])
    v = torch.randn(want.shape, generator=torch.Generator(device="cuda").manual_seed(2), device="cuda").half()
    grad, = torch.autograd.grad(got, leaf, v)
    d = torch.randn(x.shape, generator=torch.Generator(device="cuda").manual_seed(3), device="cuda").half()
    with torch.no_grad():
        assert torch.equal(neck.features(leaf), want)          # nothing records it: the kernels
    with torch.autograd.forward_ad.dual_level():
        out = torch.autograd.forward_ad.unpack_dual(neck.features(torch.autograd.forward_ad.make_dual(x, d)))
    _close(out.primal, want)
    # the same derivative from both sides; fourteen fp16 layers either way (2e-2 of the sum of magnitudes)
    a, b = float((grad.double() * d.double()).sum()), float((out.tangent.double() * v.double()).sum())
    assert abs(a - b) <= 2e-2 * float((out.tangent.double() * v.double()).abs().sum()) and out.tangent.abs().max() > 0
    neck.w["bu0_0"].requires_grad_()
    try:
        assert neck.features(x).requires_grad
    finally:
        neck.w["bu0_0"].requires_grad_(False)
    _, tangent = torch.func.jvp(neck.features, (x,), (d,))
    assert torch.equal(tangent, out.tangent)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y = neck.features(x)
    assert float((y.float() - want.float()).abs().max()) <= 0.1 * float(want.abs().max())   # fourteen layers of 2^-8
    traced = torch.jit.trace(neck.features, (x,))
    x2 = _bev(2, 10, 14, seed=8)
    _close(traced(x2), neck.features(x2))
    empty = neck(x[:0])
    assert [tuple(empty[k].shape) for k in ("box", "cls", "iou", "dir")] == [(0, 8 * 12 * 2, c) for c in (7, 1, 1, 2)]
    assert neck.features(x[:0]).shape == (0, 128, 8, 12)
    for bad in (x.float(), x[:, :64], x[0]):
        with pytest.raises(RuntimeError):
            neck.features(bad)
    host = D.Neck2D(D.random_neck_weights(), device="cpu")
    _close(host.features(x.cpu()).float(), want.float().cpu(), 2e-2)
    strided = x.transpose(2, 3)                                # neither layout
    _close(neck.features(strided), neck.features(strided.contiguous()))


def test_map_on_another_device(gpu):
    import torch

    if torch.cuda.device_count() < 2:
        pytest.skip("needs two devices")
    D, x = gpu.detector, _bev(1, 10, 14)
    want = D.Neck2D(D.random_neck_weights())(x)
    got = D.Neck2D(D.random_neck_weights(), device="cuda:1")(x.to("cuda:1"))
    for k, v in want.items():
        _close(got[k].cpu(), v.cpu())
