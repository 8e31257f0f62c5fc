"""First convolution laid out for tensor cores against the module, and the calls that must still go through it."""
import copy

import pytest
import torch
from torch import nn

from aluminum_b200.ops import stem_conv


def stem(out=64, **kw):
    return nn.Conv2d(3, out, 7, stride=2, padding=3, bias=False, **kw)


def test_on_the_cpu_it_is_the_module():
    conv, x = stem(8), torch.randn(2, 3, 9, 12)
    assert torch.equal(stem_conv(conv, x), conv(x))


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 2, 3), (1, 7, 7), (3, 9, 12), (2, 33, 30), (2, 64, 225), (4, 224, 224)])
@pytest.mark.parametrize("layout", ["rows", "channels_last", "part", "halves"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_against_64_bits(shape, layout, dtype):
    n, h, w = shape
    torch.manual_seed(h)
    x = torch.randn(n, 3, h, w, device="cuda")
    if layout == "channels_last":
        x = x.contiguous(memory_format=torch.channels_last)
    elif layout == "part":
        x = torch.randn(n, 4, h + 2, 2 * w + 1, device="cuda")[:, 1:, 1:h + 1, 1::2]
    elif layout == "halves":
        x = x.to(dtype)
    conv = stem(16 if h < 60 else 64).cuda()
    if layout != "rows":
        conv = conv.to(memory_format=torch.channels_last)
    with torch.autocast("cuda", dtype=dtype):
        y = stem_conv(conv, x)
    assert "StemConv" in y.grad_fn.name() and y.dtype == dtype and y.is_contiguous(memory_format=torch.channels_last)
    ref = copy.deepcopy(conv).double()
    with torch.no_grad():
        ref.weight.copy_(conv.weight.to(dtype).double())     # what either way multiplies
    want = ref(x.to(dtype).double())
    dy = torch.randn(want.shape, device="cuda").to(dtype)
    y.backward(dy)
    want.backward(dy.double())
    # one rounding of the result to 8 (bf16) or 11 bits, and fp32 sums
    eps = 2 ** -8 if dtype == torch.bfloat16 else 2 ** -11
    for got, exact in ((y, want), (conv.weight.grad, ref.weight.grad)):
        assert (got.double() - exact).norm() <= 0.6 * eps * exact.norm() + 1e-6 * exact.norm() and got.shape == exact.shape
    assert conv.weight.grad.stride() == conv.weight.stride()


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 8, 9), (3, 9, 12), (2, 33, 30), (2, 64, 225), (300, 16, 16)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_pixels_that_are_not_finite(shape, dtype):
    """Infinities, NaN and values beyond the 16-bit type reach the results whose windows they lie in and the weight's taps that meet them, no others."""
    n, h, w = shape
    for k, count in enumerate((1, 1, 3, 40)):
        g = torch.Generator(device="cuda").manual_seed(17 * h + k)
        x = torch.randn(n, 3, h, w, device="cuda", generator=g)
        special = torch.tensor([float("inf"), -float("inf"), float("nan"), 3.4e38], device="cuda")
        at = torch.randint(0, x.numel(), (count,), device="cuda", generator=g)
        x.view(-1)[at] = special[torch.randint(0, 4, (count,), device="cuda", generator=g)]
        conv = stem(40).cuda()
        with torch.autocast("cuda", dtype=dtype):
            y = stem_conv(conv, x)
        assert "StemConv" in y.grad_fn.name()
        ref = copy.deepcopy(conv).double()
        with torch.no_grad():
            ref.weight.copy_(conv.weight.to(dtype).double())
        want = ref(x.to(dtype).double())
        dy = torch.randn(want.shape, device="cuda", generator=g).to(dtype)
        y.backward(dy)
        want.backward(dy.double())
        eps = 2 ** -8 if dtype == torch.bfloat16 else 2 ** -11
        for got, exact in ((y, want), (conv.weight.grad, ref.weight.grad)):
            if dtype == torch.float16:     # (the library's convolutions of channels-last fp16 images, the module's too, give 0 for minus infinity)
                got = torch.where((exact == -float("inf")) & (got == 0), exact, got.double())
            ok = exact.isfinite()
            assert torch.equal(got.isfinite(), ok) and torch.equal(got.isnan(), exact.isnan()) and torch.equal(got == float("inf"), exact == float("inf"))
            got, exact = got[ok].double(), exact[ok]
            assert (got - exact).norm() <= 0.6 * eps * exact.norm() + 1e-6 * exact.norm()


@pytest.mark.gpu
def test_second_derivative_and_a_weight_that_changes_before_the_backward():
    x, conv = torch.randn(2, 3, 18, 20, device="cuda"), stem(8).cuda()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        a, b = stem_conv(conv, x), conv(x)
    ga, = torch.autograd.grad((a.float() ** 2).sum(), conv.weight, create_graph=True)
    gb, = torch.autograd.grad((b.float() ** 2).sum(), conv.weight, create_graph=True)
    assert torch.allclose(ga, gb, rtol=2e-2, atol=2e-2 * gb.abs().max().item())
    sa, sb = (torch.autograd.grad(g.square().sum(), conv.weight)[0] for g in (ga, gb))
    assert (sa - sb).norm() <= 3e-2 * sb.norm()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y = stem_conv(conv, x)
    with torch.no_grad():
        conv.weight.add_(1)
    y.sum().backward()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        want, = torch.autograd.grad(conv(x).sum(), conv.weight)     # (the weight is no part of it)
    assert (conv.weight.grad - want).norm() <= 2 ** -7 * want.norm()   # two results rounded to 8 bits


@pytest.mark.gpu
def test_calls_that_stay_with_the_module():
    x, conv = torch.randn(2, 3, 20, 20, device="cuda"), stem(16).cuda()

    def taken(conv, x, dtype=torch.bfloat16):
        with torch.autocast("cuda", dtype=dtype):
            y, want = stem_conv(conv, x), conv(x)
        if y.grad_fn is not None and "StemConv" in y.grad_fn.name():
            return True
        assert torch.equal(y, want)
        return False
    assert taken(conv, x)
    assert not taken(conv, x.clone().requires_grad_())
    assert not taken(conv.eval(), x)
    conv.train()
    with torch.no_grad():
        assert not taken(conv, x)
    with torch.inference_mode():
        assert not taken(conv, x)
    assert torch.equal(stem_conv(conv, x), conv(x)) and "StemConv" not in stem_conv(conv, x).grad_fn.name()   # no autocast
    assert not taken(conv, x.half())                                   # of another type than autocast's
    for other in (nn.Conv2d(3, 16, 7, stride=2, padding=3), nn.Conv2d(3, 16, 7, stride=2, padding=2, bias=False), nn.Conv2d(3, 16, 5, stride=2, padding=3, bias=False),
                  nn.Conv2d(3, 16, 7, padding=3, bias=False), stem(12), stem(16, padding_mode="circular"), stem(16).requires_grad_(False)):
        assert not taken(other.cuda(), x)
    hooked = stem(16).cuda()
    hooked.register_forward_hook(lambda m, i, o: o * 2)
    assert not taken(hooked, x)
    compiled = torch.compile(lambda c, v: stem_conv(c, v), backend="eager", fullgraph=True)
    assert compiled(conv, x).shape == (2, 16, 10, 10)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_weights_cast_together(dtype):
    """Values, gradients and their layouts of autocast's casts one by one; sizes around a tile; a weight that goes unused."""
    from aluminum_b200.ops.convolution import cast_weights, convolve
    torch.manual_seed(0)
    cl = dict(memory_format=torch.channels_last)
    convs = [nn.Conv2d(16, 32, 3, padding=1, bias=False), nn.Conv2d(32, 128, 1, bias=False), nn.Conv2d(128, 7, 3, stride=2, bias=False),
             nn.Conv2d(16, 1, 1, bias=False)]
    convs = [c.cuda().to(**cl) for c in convs]
    x = torch.randn(2, 16, 10, 10, device="cuda").to(dtype).contiguous(**cl)

    def run(together):
        net = [copy.deepcopy(c) for c in convs]
        with torch.autocast("cuda", dtype=dtype):
            w = cast_weights(net, x) if together else [None] * 4
            y = x
            for c, v in zip(net[:3], w):
                assert not together or (v.dtype == dtype and torch.equal(v, c.weight.to(dtype)) and v.stride() == c.weight.stride())
                y = convolve(c, y, v)
            y.float().square().mean().backward()
        return [y] + [c.weight.grad for c in net]
    for a, b in zip(run(True), run(False)):
        assert (a is None and b is None) or (torch.allclose(a, b, rtol=1e-2, atol=1e-4) and a.stride() == b.stride() and a.dtype == b.dtype)
    with torch.autocast("cuda", dtype=dtype):
        def second(w):
            g, = torch.autograd.grad(convolve(convs[0], x, w).float().square().mean(), convs[0].weight, create_graph=True)
            assert g.dtype == torch.float32
            return torch.autograd.grad(g.square().sum(), convs[0].weight)[0]
        a, b = second(cast_weights(convs[:1], x)[0]), second(None)
        assert b.norm() > 0 and (a - b).norm() <= 1e-2 * b.norm()
        hooked, biased, frozen = (copy.deepcopy(convs[0]) for _ in range(3))
        hooked.register_forward_pre_hook(lambda *a: None)
        biased.bias = nn.Parameter(torch.zeros(32, device="cuda"))
        frozen.weight.requires_grad_(False)
        for other in (hooked, biased, frozen):
            assert cast_weights([convs[0], other], x) is None
        assert cast_weights(convs, x.float()) is None
        with torch.no_grad():
            assert cast_weights(convs, x) is None
    assert cast_weights(convs, x) is None     # no autocast


@pytest.mark.gpu
@pytest.mark.parametrize("case", ["own", "hook", "fp32", "other", "evaluation", "wide"])
def test_images_are_laid_out_where_the_first_convolution_does_not(case, monkeypatch):
    """The trainer's promise of channels-last images holds for every first convolution but the one that takes any layout."""
    from aluminum_b200.models import resnet
    from aluminum_b200.parallel import DataParallel, Trainer
    net, seen = resnet.ResNet((1, 1, 1, 1), 10, width=16).cuda(), []
    stem_conv = resnet.stem_conv

    def watched(conv, x):
        seen.append(x.is_contiguous(memory_format=torch.channels_last))
        return stem_conv(conv, x)
    monkeypatch.setattr(resnet, "stem_conv", watched)
    if case == "hook":
        net.conv1.register_forward_pre_hook(lambda *a: None)
    elif case == "other":
        net.conv1 = nn.Sequential(nn.Conv2d(3, 16, 3, stride=2, padding=1, bias=False)).cuda()
    elif case == "evaluation":
        net.conv1.eval()
    trainer = Trainer(DataParallel(net, None, lr=0.01), autocast_dtype=None if case == "fp32" else torch.bfloat16)
    x = torch.randn(2, 3, 32, 704 if case == "wide" else 40, device="cuda")
    trainer.step_device(x, torch.tensor([1, 2], device="cuda"))
    assert seen == [case != "own"]
