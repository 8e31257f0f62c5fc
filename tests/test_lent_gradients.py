"""The optimizer step on gradients where backward left them: bit for bit the step on the flat gradient, whatever form they come in."""
import copy

import pytest
import torch
from torch import nn

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def al():
    import aluminum_b200 as al
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    al.init()
    return al


@pytest.fixture(autouse=True)
def repeatable(monkeypatch):
    monkeypatch.setattr(torch.backends.cudnn, "deterministic", True)


class Odd(torch.autograd.Function):
    """Identity on a parameter whose gradient comes expanded, transposed or off its 16 bytes."""

    @staticmethod
    def forward(ctx, p, kind):
        ctx.kind = kind
        return p.clone()

    @staticmethod
    def backward(ctx, g):
        if ctx.kind == "expanded":
            return g.flatten()[0].expand(g.shape), None
        if ctx.kind == "transposed":
            return g.t().contiguous().t(), None
        flat = torch.empty(g.numel() + 1, device=g.device)[1:]
        return flat.copy_(g.flatten()).view(g.shape), None


class Net(nn.Module):
    def __init__(self):
        super().__init__()
        self.conv = nn.Conv2d(3, 8, 3)
        self.bn = nn.BatchNorm2d(8)
        self.odd = nn.ParameterList([nn.Parameter(torch.randn(7, 5)) for _ in range(3)])
        self.unused = nn.Parameter(torch.randn(13))
        self.wide = nn.Linear(8 * 36, 1029)      # more than a tile, and a remainder

    def forward(self, x):
        x = self.wide(self.bn(self.conv(x)).flatten(1))
        for p, kind in zip(self.odd, ("expanded", "transposed", "shifted")):
            x = x + Odd.apply(p, kind).square().sum()
        return x


class Native(Net):
    """The same without functions written in Python: gradients that are parts of one tensor, off their 16 bytes among them."""

    def forward(self, x):
        x = self.wide(self.bn(self.conv(x)).flatten(1))
        return x + torch.cat([p.flatten() for p in self.odd]).square().sum()


def pair(net, **kw):
    from aluminum_b200.parallel import DataParallel, Trainer
    made = []
    for _ in range(2):
        dp = DataParallel(copy.deepcopy(net).cuda().to(memory_format=torch.channels_last), None, lr=0.05, momentum=0.9, weight_decay=1e-3, **kw)
        made.append((Trainer(dp, autocast_dtype=None), dp))
    made[1][1].step = lambda d=made[1][1]: type(d).step(d)     # a step of the instance's own: by way of the flat gradient
    return made


@pytest.mark.parametrize("net", [Net, Native])
def test_equals_the_step_on_the_flat_gradient(net):
    torch.manual_seed(0)
    (a, da), (b, db) = pair(net())
    x, y = torch.randn(6, 3, 8, 8, device="cuda"), torch.randint(0, 1029, (6,), device="cuda")
    for k in range(4):
        if k == 2:     # gradients that a backward of the caller's own has left
            for dp in (da, db):
                dp(x).square().mean().backward()
        la, lb = a.step_device(x, y), b.step_device(x, y)
        assert torch.equal(la, lb)
        for u, v in ((da.flat_param, db.flat_param), (da.flat_mom, db.flat_mom)):
            assert torch.equal(u, v)
        assert not da.flat_grad.any() and da.steps == db.steps and da.launches == db.launches
        for p, view in zip(da._params, da._grad_views):
            assert p.grad is view
    da.lr = db.lr = 0.5
    assert torch.equal(a.step_device(x, y), b.step_device(x, y)) and torch.equal(da.flat_param, db.flat_param)


def lend(dp, x):
    """A backward on lent gradients; False: they were not lent."""
    from aluminum_b200 import _lib
    loss = dp(x).square().mean()
    if not _lib.calls().lend_gradients(loss, dp._params, dp._grad_views):
        return False
    assert all(p.grad is None for p in dp._params)
    loss.backward()
    return True


def test_which_forms_reach_the_optimizer():
    torch.manual_seed(0)
    (_, da), (_, db) = pair(Native())
    x = torch.randn(6, 3, 8, 8, device="cuda")
    assert lend(da, x) and not lend(pair(Net())[0][1], x)
    assert any(p.grad is not None and p.grad.data_ptr() % 16 for p in da._params) and any(p.grad is None for p in da._params)


@pytest.mark.parametrize("kind", ["post_accumulate", "tensor", "module", "node", "activation"])
def test_what_runs_in_the_backward_finds_the_gradients(kind):
    """Clipping by way of the flat gradient or of a gradient held from before: lent gradients would be somewhere else."""
    torch.manual_seed(0)
    net = nn.Sequential(nn.Conv2d(3, 8, 3), nn.Flatten(), nn.Linear(8 * 36, 10))
    (a, da), (b, db) = pair(net)
    x, y, keep = torch.randn(6, 3, 8, 8, device="cuda"), torch.randint(0, 10, (6,), device="cuda"), []
    for dp in (da, db):
        held, (conv, _, linear) = [p.grad for p in dp._params], dp.module

        def clip(*_, dp=dp, held=held):
            dp.flat_grad.mul_(0.25)
            held[-1].add_(0.125)
        if kind == "post_accumulate":
            linear.bias.register_post_accumulate_grad_hook(clip)
        elif kind == "tensor":
            conv.bias.register_hook(clip)
        elif kind == "module":
            linear.register_full_backward_hook(clip)
        elif kind == "node":
            keep.append(linear.bias.expand_as(linear.bias).grad_fn.next_functions[0][0])
            keep[-1].register_hook(clip)
        else:
            conv.register_forward_hook(lambda m, i, o, clip=clip: o.register_hook(clip) and None)
    for _ in range(2):
        a.step_device(x, y)
        b.step_device(x, y)
    assert torch.equal(da.flat_param, db.flat_param) and torch.equal(da.flat_mom, db.flat_mom)


def test_a_gradient_that_is_its_view_counts_once():
    from aluminum_b200 import _lib
    torch.manual_seed(0)
    (_, da), (_, db) = pair(Native())
    x = torch.randn(6, 3, 8, 8, device="cuda")
    assert lend(da, x)
    for k, (p, view) in enumerate(zip(da._params, da._grad_views)):
        if k % 2 and p.grad is not None:
            view.copy_(p.grad)
            p.grad = view.detach() if k % 4 == 1 else view
    _lib.calls().step_on_lent(da._params, da._grad_views, da.flat_param, da.flat_mom, da.flat_grad, 0.05, 0.9, 1e-3, True)
    db(x).square().mean().backward()
    db.step()
    assert torch.equal(da.flat_param, db.flat_param) and torch.equal(da.flat_mom, db.flat_mom) and not da.flat_grad.any()
    assert all(p.grad is v for p, v in zip(da._params, da._grad_views))


def test_a_step_that_is_refused_keeps_the_gradients():
    from aluminum_b200 import _lib
    torch.manual_seed(0)
    (_, da), (_, db) = pair(Native())
    x, before = torch.randn(6, 3, 8, 8, device="cuda"), da.flat_param.clone()
    assert lend(da, x)
    with pytest.raises(_lib.AlError, match="not of the form"):     # views that do not begin on 16 bytes of the flat buffer
        _lib.calls().step_on_lent(da._params, da._grad_views, da.flat_param, da.flat_mom, da.flat_grad[1:], 0.05, 0.9, 1e-3, True)
    db(x).square().mean().backward()
    assert torch.equal(da.flat_param, before) and torch.equal(da.flat_grad, db.flat_grad)
    assert all(p.grad is v for p, v in zip(da._params, da._grad_views))


def test_a_backward_on_lent_gradients_that_fails_keeps_what_it_has():
    torch.manual_seed(0)
    (_, da), _ = pair(Native())
    net = da.module
    s = net.conv(torch.randn(6, 3, 8, 8, device="cuda")).square()
    s.sum().backward()
    before = [v.clone() for v in da._grad_views]
    with pytest.raises(RuntimeError, match="second time"):     # behind the last layers, whose gradients are there by then
        da.backward_and_step(net.wide(net.bn(s).flatten(1)).square().mean())
    assert da.steps == 0 and all(p.grad is v for p, v in zip(da._params, da._grad_views))
    for p, was in zip(da._params, before):
        assert torch.equal(p.grad, was) != (p is net.wide.weight or p is net.wide.bias or p is net.bn.weight or p is net.bn.bias)


def test_a_backward_that_fails_keeps_what_it_has():
    torch.manual_seed(0)
    (a, da), _ = pair(Net())
    x, y = torch.randn(6, 3, 8, 8, device="cuda"), torch.randint(0, 1029, (6,), device="cuda")
    before, handle = da.flat_param.clone(), da.module.conv.weight.register_hook(lambda g: 1 / 0)
    with pytest.raises(ZeroDivisionError):
        a.step_device(x, y)
    handle.remove()
    assert torch.equal(da.flat_param, before) and da.steps == 0
    assert all(p.grad is v for p, v in zip(da._params, da._grad_views)) and da.flat_grad.any()
    da.module.conv.weight.grad = None     # not its view: the step is the one by way of the flat gradient, which this parameter has left
    a.step_device(x, y)
    assert da.steps == 1 and da.module.conv.weight.grad is not None and da.module.bn.weight.grad is not None


@pytest.mark.parametrize("sizes", [[1], [3, 4, 5], [4095, 4096, 4097, 1], [8192 + 17], [5] * 700])
@pytest.mark.parametrize("first", [True, False])
def test_kernel_against_the_flat_step(sizes, first):
    """Tile edges, remainders, tensors without a gradient, more tensors than a launch takes."""
    import ctypes as C
    from aluminum_b200 import _lib
    from aluminum_b200.ops import sgd_momentum_step
    at = [0]
    for n in sizes:
        at.append(at[-1] + (n + 3) // 4 * 4)
    g = torch.Generator(device="cuda").manual_seed(len(sizes))
    p, m, f = (torch.randn(at[-1], generator=g, device="cuda") for _ in range(3))
    inside = torch.zeros(at[-1], dtype=torch.bool, device="cuda")
    for n, o in zip(sizes, at):
        inside[o:o + n] = True
    f[~inside] = 0
    grads = [torch.randn(n, generator=g, device="cuda") if k % 5 != 3 else None for k, n in enumerate(sizes)]
    want = [t.clone() for t in (p, m, f)]
    for t, n, o in zip(grads, sizes, at):
        if t is not None:
            want[2][o:o + n] += t
    sgd_momentum_step(want[0], want[1], want[2], 0.1, 0.9, 1e-2, 1.0, first_step=first, zero_grad=True)
    k = len(sizes)
    ptr = lambda t: C.c_void_p(t.data_ptr() if t is not None else None)
    lib = _lib.load()
    _lib.check(lib.al_sgd_momentum_from(ptr(p), ptr(m), ptr(f), (C.c_void_p * k)(*[t.data_ptr() if t is not None else None for t in grads]),
                                        (C.c_size_t * k)(*at[:-1]), (C.c_size_t * k)(*sizes), k, C.c_float(0.1), C.c_float(0.9), C.c_float(1e-2),
                                        C.c_float(1.0), int(first), C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    for got, exact in zip((p, m, f), want):
        assert torch.equal(got[inside], exact[inside])
    assert lib.al_sgd_momentum_from(ptr(p), ptr(m), ptr(f), (C.c_void_p * 1)(p.data_ptr() + 4), (C.c_size_t * 1)(0), (C.c_size_t * 1)(1), 1, C.c_float(0.1),
                                    C.c_float(0.9), C.c_float(0), C.c_float(1), 0, C.c_void_p(0)) != 0     # (not on 16 bytes: refused)
