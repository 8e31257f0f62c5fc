"""Fused training batch norm (+ residual, + ReLU) against the same operation in 64 bits, and the calls that must still
go through the modules."""
import copy

import pytest
import torch
from torch import nn

from aluminum_b200.ops import batch_norm_act, max_pool


def reference(bn, x, residual, relu, dy):
    """Outputs, gradients and running statistics in 64 bits."""
    bn = copy.deepcopy(bn).double()
    x = x.detach().double().requires_grad_()
    res = residual.detach().double().requires_grad_() if residual is not None else None
    y = bn(x)
    if res is not None:
        y = y + res
    if relu:
        y = y.relu()
    y.backward(dy.double())
    return y, x.grad, res.grad if res is not None else None, bn.weight.grad, bn.bias.grad, bn.running_mean, bn.running_var


def rel(a, b):
    return ((a.double() - b).norm() / b.norm().clamp_min(1e-30)).item()


# channels: one column, a part of a warp's columns, whole warps and a ragged tile; rows around a thread's, a CTA's and the grid's share
SHAPES = [(2, 8, 1, 1), (3, 24, 5, 7), (2, 64, 33, 31), (1, 264, 9, 9), (5, 2048, 7, 7), (24, 256, 56, 56), (9, 64, 112, 112)]


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("relu,res", [(True, False), (True, True), (False, False), (False, True)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_against_64_bits(shape, relu, res, dtype):
    torch.manual_seed(sum(shape))
    cl = dict(memory_format=torch.channels_last)
    n, c, h, w = shape
    bn = nn.BatchNorm2d(c).cuda()
    nn.init.uniform_(bn.weight, 0.5, 1.5)
    nn.init.uniform_(bn.bias, -1, 1)
    offset = torch.linspace(-20, 20, c, device="cuda").view(1, c, 1, 1)   # means well away from 0: deviations, not squares, are summed
    make = lambda: torch.randn(shape, device="cuda")
    x = (make() + offset).to(dtype).contiguous(**cl).requires_grad_()
    residual = make().to(dtype).contiguous(**cl).requires_grad_() if res else None
    dy = make().to(dtype).contiguous(**cl)
    want = reference(bn, x, residual, relu, dy)
    y = batch_norm_act(bn, x, nn.ReLU(inplace=True) if relu else None, residual)
    assert "BatchNormAct" in y.grad_fn.name()
    y.backward(dy)
    # One rounding to 16 bits on the way out.  Gradients behind a ReLU: inputs reach 25, so sums in 32 bits are off by
    # up to 25 * 1.5 * 2^-23 = 4.5e-6 in front of the ReLU; with a density of 0.4 around 0 that is 3.6e-6 of the
    # elements whose gradient may pass or stop, and the square root of it in the norm.
    flips = 1.9e-3 if relu else 0.0
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    small = n * h * w < 64        # few rows: the gradient of x is a difference of nearly equal terms
    assert rel(y, want[0]) < eps
    assert rel(x.grad, want[1]) < (0.5 if small else 4 * eps + flips)
    if res:
        assert rel(residual.grad, want[2]) < eps + flips
    assert rel(bn.weight.grad, want[3]) < (1e-2 if small else 4 * eps)
    assert rel(bn.bias.grad, want[4]) < 4 * eps
    assert rel(bn.running_mean, want[5]) < 1e-6
    assert rel(bn.running_var, want[6]) < 1e-5
    assert int(bn.num_batches_tracked) == 1


@pytest.mark.gpu
def test_nan_infinity_and_second_derivative():
    cl = dict(memory_format=torch.channels_last)
    bn = nn.BatchNorm2d(16).cuda()
    x = torch.randn(2, 16, 4, 4, device="cuda").bfloat16().contiguous(**cl)
    x[0, 3, 1, 1] = float("nan")
    x[1, 5, 0, 0] = float("inf")
    y = batch_norm_act(bn, x, nn.ReLU())
    want = torch.relu(copy.deepcopy(bn)(x))
    assert torch.equal(torch.isnan(y), torch.isnan(want))
    x = torch.randn(2, 16, 4, 4, device="cuda").bfloat16().contiguous(**cl).requires_grad_()
    got = []
    for f in (lambda: batch_norm_act(bn, x, nn.ReLU()), lambda: torch.relu(bn(x))):
        g, = torch.autograd.grad(f().float().square().sum(), x, create_graph=True)
        got.append(torch.autograd.grad(g.float().square().sum(), x)[0].double())
    assert rel(got[0], got[1]) < 5e-2   # a chain of 16-bit operations, in another order


@pytest.mark.gpu
def test_calls_that_stay_with_the_modules():
    cl = dict(memory_format=torch.channels_last)
    x = torch.randn(2, 16, 4, 4, device="cuda").bfloat16().contiguous(**cl)
    relu = nn.ReLU()
    seen = []
    hooked = nn.BatchNorm2d(16).cuda()
    hooked.register_forward_hook(lambda *a: seen.append(1))
    batch_norm_act(hooked, x, relu)
    assert seen
    bn = nn.BatchNorm2d(16).cuda()
    for bad in (x.float(), x.contiguous(), x[:, :, ::2]):
        got = batch_norm_act(copy.deepcopy(bn), bad, relu)
        assert torch.equal(got, relu(copy.deepcopy(bn)(bad)))
    assert torch.equal(batch_norm_act(copy.deepcopy(bn).eval(), x, relu), relu(copy.deepcopy(bn).eval()(x)))
    with pytest.raises(ValueError):
        batch_norm_act(bn, x[:1, :, :1, :1].contiguous(**cl), relu)


def test_cpu_and_scripted_block():
    from aluminum_b200.models.resnet import Bottleneck
    bn, x = nn.BatchNorm2d(8), torch.randn(2, 8, 3, 3)
    assert torch.equal(batch_norm_act(copy.deepcopy(bn), x, nn.ReLU(), x), torch.relu(bn(x) + x))
    block = Bottleneck(16, 4)
    scripted = torch.jit.script(copy.deepcopy(block))
    x = torch.randn(2, 16, 5, 5)
    assert torch.allclose(block(x), scripted(x), atol=1e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("k,stride,pad", [(3, 2, 1), (2, 2, 0), (3, 1, 1), (5, 3, 2), (1, 1, 0), (2, 3, 1)])
@pytest.mark.parametrize("shape", [(2, 8, 5, 5), (3, 24, 13, 7), (2, 64, 112, 112)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_max_pool(k, stride, pad, shape, dtype):
    torch.manual_seed(k)
    cl = dict(memory_format=torch.channels_last)
    pool = nn.MaxPool2d(k, stride, pad)
    x = torch.randint(-9, 9, shape, device="cuda").to(dtype).contiguous(**cl).requires_grad_()   # many equal values
    y = max_pool(pool, x)
    assert "MaxPool" in y.grad_fn.name() and "MaxPool2D" not in y.grad_fn.name()
    xr = x.detach().double().contiguous().requires_grad_()
    want = pool(xr)
    assert torch.equal(y.double(), want)
    dy = torch.randint(-3, 4, want.shape, device="cuda").to(dtype)   # sums of a few small integers are exact
    y.backward(dy)
    want.backward(dy.double())
    assert torch.equal(x.grad.double(), xr.grad)
    g, = torch.autograd.grad((max_pool(pool, x).float() ** 2).sum(), x, create_graph=True)
    assert torch.equal(torch.autograd.grad(g.float().sum(), x)[0].double() != 0, torch.autograd.grad((pool(xr) ** 2).sum(), xr)[0] * 0 +
                       torch.autograd.grad(torch.autograd.grad((pool(xr) ** 2).sum(), xr, create_graph=True)[0].sum(), xr)[0] != 0)


@pytest.mark.gpu
def test_max_pool_nan_and_module_calls():
    cl = dict(memory_format=torch.channels_last)
    x = torch.randn(2, 8, 6, 6, device="cuda").bfloat16().contiguous(**cl)
    x[0, 1, 2, 3] = float("nan")
    pool = nn.MaxPool2d(3, 2, 1)
    assert torch.equal(torch.isnan(max_pool(pool, x)), torch.isnan(pool(x)))
    for other in (nn.MaxPool2d(3, 2, 1, ceil_mode=True), nn.MaxPool2d((3, 2), 2), nn.MaxPool2d(2, dilation=2)):
        assert torch.equal(max_pool(other, x.nan_to_num()), other(x.nan_to_num()))
    assert torch.equal(max_pool(pool, x.float().nan_to_num()), pool(x.float().nan_to_num()))
    with pytest.raises(RuntimeError):
        max_pool(nn.MaxPool2d(3, 1, 2), x)


@pytest.mark.gpu
@pytest.mark.parametrize("hooks", ["pinned", "permuted", "unaligned"])
def test_saved_tensors_in_another_layout(hooks):
    """Saved-tensor hooks give back the values, not always the layout: gradients are those without hooks, bit for bit."""
    def unaligned(t):
        flat = torch.empty(t.numel() + 1, device=t.device, dtype=t.dtype)[1:]
        return torch.as_strided(flat, t.shape, t.stride()).copy_(t)
    context = {"pinned": lambda: torch.autograd.graph.save_on_cpu(pin_memory=True),   # comes back contiguous, not channels-last
               "permuted": lambda: torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t.contiguous().clone()),
               "unaligned": lambda: torch.autograd.graph.saved_tensors_hooks(lambda t: t, unaligned)}[hooks]
    torch.manual_seed(3)
    cl = dict(memory_format=torch.channels_last)
    bn, pool = nn.BatchNorm2d(24).cuda(), nn.MaxPool2d(3, 2, 1)
    x0, r0 = (torch.randn(3, 24, 9, 7, device="cuda").bfloat16().contiguous(**cl) for _ in range(2))
    got = []
    for hooked in (False, True):
        b = copy.deepcopy(bn)
        x, r = x0.clone().requires_grad_(), r0.clone().requires_grad_()
        if hooked:
            with context():
                y = max_pool(pool, batch_norm_act(b, x, nn.ReLU(), r))
        else:
            y = max_pool(pool, batch_norm_act(b, x, nn.ReLU(), r))
        assert "MaxPool" in y.grad_fn.name() and "MaxPool2D" not in y.grad_fn.name()
        y.backward(torch.linspace(-1, 1, y.numel(), device="cuda").view(y.shape).bfloat16().contiguous(**cl))
        got.append([x.grad, r.grad, b.weight.grad, b.bias.grad])
    assert all(torch.equal(u, v) for u, v in zip(*got))


@pytest.mark.parametrize("training", [True, False])
def test_compiled_model_stays_one_graph(training):
    from aluminum_b200.models.resnet import ResNet
    torch.manual_seed(0)
    model, x = ResNet((1, 1, 1, 1), num_classes=10).train(training), torch.randn(2, 3, 32, 32)
    want = copy.deepcopy(model)(x)
    torch._dynamo.reset()
    got = torch.compile(copy.deepcopy(model), fullgraph=True, backend="eager")(x)   # raises at a graph break
    assert torch.allclose(got, want, atol=1e-5)


def test_parameters_of_another_length_or_kind_go_to_the_module():
    from aluminum_b200.ops import activations

    class Wrapped(torch.Tensor):
        pass
    assert activations._parameter_ok(torch.zeros(8), 8, -1) and activations._parameter_ok(nn.Parameter(torch.zeros(8)), 8, -1)
    for other in (torch.zeros(7), torch.zeros(16), torch.zeros(8).double(), torch.zeros(8).as_subclass(Wrapped), None):
        assert not activations._parameter_ok(other, 8, -1)


def test_forward_of_the_instances_own():
    from aluminum_b200.models.resnet import Shortcut
    from aluminum_b200.ops import activations
    for m in (nn.BatchNorm2d(8), nn.ReLU(), nn.MaxPool2d(2)):
        assert activations._bare(m)
        m.forward = m.forward
        assert not activations._bare(m)
    x = torch.randn(2, 4, 3, 3)
    parts = [nn.Conv2d(4, 8, 1), nn.BatchNorm2d(8), nn.ReLU()]
    for n in (1, 2, 3):
        assert torch.equal(Shortcut(*copy.deepcopy(parts[:n]))(x), nn.Sequential(*copy.deepcopy(parts[:n]))(x))


@pytest.mark.gpu
def test_stopped_infinite_gradient_in_a_graph_of_the_backward():
    cl = dict(memory_format=torch.channels_last)
    torch.manual_seed(5)
    bn = nn.BatchNorm2d(16).cuda()
    x = torch.randn(2, 16, 6, 6, device="cuda").bfloat16().contiguous(**cl).requires_grad_()
    y = batch_norm_act(bn, x, nn.ReLU())
    dy = torch.where(y > 0, torch.randn_like(y), float("inf")).detach()
    g, = torch.autograd.grad(y, x, dy, retain_graph=True)
    h, = torch.autograd.grad(y, x, dy, create_graph=True)
    assert torch.isfinite(g).all() and rel(h.detach(), g.double()) < 1e-2


@pytest.mark.gpu
@pytest.mark.parametrize("rows,channels", [(2, 8), (3, 64), (33, 264), (129, 2048), (1025, 520), (592 * 128 + 5, 64), (592 * 128 - 1, 72)])
@pytest.mark.parametrize("offset", [0.0, 64.0])
def test_statistics_at_the_edges_of_tiles_and_partials(rows, channels, offset):
    """One row more or less than threads, tiles and CTAs have; means far from 0.  With a momentum of 1 the running statistics are the batch's."""
    from aluminum_b200.ops import batch_norm_act
    torch.manual_seed(rows)
    x = (torch.randn(1, channels, rows, 1, device="cuda") + offset).bfloat16().contiguous(memory_format=torch.channels_last)
    x[0, :, 0] += 3   # where the sums begin
    bn = nn.BatchNorm2d(channels, momentum=1.0).cuda()
    x.requires_grad_()
    y = batch_norm_act(bn, x, nn.ReLU())
    assert "BatchNormAct" in y.grad_fn.name()
    v = x.detach().double()[0, :, :, 0]
    mean, var = v.mean(1), v.var(1)
    # fp32 sums of deviations: a few roundings of the deviations' size, and one of the mean's
    assert ((bn.running_mean - mean).abs() <= 2e-6 * (var.sqrt() + 1) + 1.2e-7 * mean.abs()).all()
    assert ((bn.running_var - var).abs() <= 5e-6 * var + 1e-12).all()
    y.backward(torch.ones_like(y))
    passes = (y.detach() > 0).double()[0, :, :, 0]
    assert ((bn.bias.grad - passes.sum(1)).abs() <= 1e-6 * rows).all()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("h,w", [(1, 1), (1, 2), (2, 1), (3, 3), (2, 7), (8, 9), (15, 16)])
def test_pooling_by_three_every_two(h, w, dtype):
    """Windows cut by every border, with equal values, both zeros, infinities and NaN among them: value and place of the module's winner."""
    cl = dict(memory_format=torch.channels_last)
    pool = nn.MaxPool2d(3, 2, 1)
    g = torch.Generator(device="cuda").manual_seed(h * 20 + w)
    special = torch.tensor([0.0, -0.0, 1.0, -1.0, 2.0, float("inf"), -float("inf"), -float("inf"), float("nan"), -3.0], device="cuda")
    for most in (5, 8, 10):   # without infinities and NaN, without NaN, with all
        x = special[torch.randint(0, most, (3, 16, h, w), generator=g, device="cuda")].to(dtype).contiguous(**cl).requires_grad_()
        y = max_pool(pool, x)
        assert "MaxPool" in y.grad_fn.name() and "MaxPool2D" not in y.grad_fn.name()
        xr = x.detach().float().contiguous().requires_grad_()
        want = pool(xr)
        assert torch.equal(y.float().nan_to_num(nan=99.0), want.nan_to_num(nan=99.0))
        dy = torch.randint(-3, 4, want.shape, generator=g, device="cuda").to(dtype)
        y.backward(dy)
        want.backward(dy.float())
        assert torch.equal(x.grad.float(), xr.grad)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(2, 8, 1, 1), (3, 24, 5, 7), (2, 264, 33, 31), (5, 2048, 7, 7), (24, 64, 56, 56)])
@pytest.mark.parametrize("relu,res", [(True, True), (True, False), (False, True), (False, False)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_output_used_twice(shape, relu, res, dtype):
    """The two gradients added by the kernel: bit for bit what the framework's addition of them gives."""
    from aluminum_b200.ops import batch_norm_act_twice
    torch.manual_seed(shape[1])
    cl = dict(memory_format=torch.channels_last)
    rand = lambda: torch.randn(shape, device="cuda").to(dtype).contiguous(**cl)
    bn, x0, r0, a, b = nn.BatchNorm2d(shape[1]).cuda(), rand(), rand(), rand(), rand()
    act = nn.ReLU() if relu else None

    def run(use):
        m, x, r = copy.deepcopy(bn), x0.clone().requires_grad_(), r0.clone().requires_grad_()
        use(m, x, r if res else None)
        return [x.grad, m.weight.grad, m.bias.grad, m.running_mean] + ([r.grad] if res else [])

    def twice(m, x, r):
        y, same = batch_norm_act_twice(m, x, act, r)
        assert "BatchNormAct" in y.grad_fn.name() and same.data_ptr() == y.data_ptr() and same.grad_fn is y.grad_fn
        torch.autograd.backward([y, same], [a, b])

    def once(m, x, r):
        batch_norm_act(m, x, act, r).backward(a + b)
    assert all(torch.equal(u, v) for u, v in zip(run(twice), run(once)))
    for used in (0, 1):   # only one of the two used
        def single(m, x, r):
            batch_norm_act_twice(m, x, act, r)[used].backward(a)
        assert all(torch.equal(u, v) for u, v in zip(run(single), run(lambda m, x, r: batch_norm_act(m, x, act, r).backward(a))))

    def graph(pair):
        def use(m, x, r):
            outputs, gradients = (batch_norm_act_twice(m, x, act, r), (a, b)) if pair else ((batch_norm_act(m, x, act, r),), (a + b,))
            gx, = torch.autograd.grad(outputs, [x], gradients, create_graph=True)
            (gx.float().square().mean() + outputs[0].float().mean()).backward()
        return use
    for u, v in zip(run(graph(True)), run(graph(False))):
        assert torch.equal(u.nan_to_num(7.0), v.nan_to_num(7.0))


@pytest.mark.gpu
def test_network_block_by_block():
    """The network's own loop over its blocks: the gradients of calling the stages, to what the order of one addition is worth;
    hooks on a stage or a block are called."""
    from aluminum_b200.models.resnet import ResNet
    torch.manual_seed(0)
    net = ResNet((2, 2, 1, 1), 10, width=16).cuda().to(memory_format=torch.channels_last)
    for m in net.modules():
        if isinstance(m, nn.BatchNorm2d):
            nn.init.uniform_(m.weight, 0.5, 1.5)
    x = torch.randn(4, 3, 64, 64, device="cuda")

    def grads(net):
        with torch.autocast("cuda", dtype=torch.bfloat16):
            net(x).float().square().mean().backward()
        return [p.grad for p in net.parameters()]
    own, called, seen = copy.deepcopy(net), copy.deepcopy(net), []
    for stage in (called.layer1, called.layer3):
        stage.register_forward_hook(lambda *a: seen.append(1))
    for u, v in zip(grads(own), grads(called)):
        assert rel(u, v.double()) < 2e-2
    assert len(seen) == 2
    called = copy.deepcopy(net)
    called.layer2[1].register_forward_pre_hook(lambda *a: seen.append(1))
    grads(called)
    assert len(seen) == 3


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["conv1", "downsample", "shortcut", "convolution"])
def test_modules_that_write_to_a_blocks_input(where):
    """A module put in front of a block's first convolution or of its shortcut may work in place: both then see what it made."""
    from aluminum_b200.models.resnet import ResNet, Shortcut
    torch.manual_seed(0)
    net = ResNet((2, 1, 1, 1), 10, width=16).cuda().to(memory_format=torch.channels_last)
    for m in net.modules():
        if isinstance(m, nn.BatchNorm2d):
            nn.init.uniform_(m.weight, 0.5, 1.5)

    class Gated(nn.Conv2d):
        def forward(self, x):
            return super().forward(x.mul_(0.5))
    block = net.layer1[1]
    if where == "conv1":
        block.conv1 = nn.Sequential(nn.Hardswish(inplace=True), block.conv1)
    elif where == "downsample":
        block.downsample = nn.Hardswish(inplace=True)
    elif where == "shortcut":
        block = net.layer2[0]
        block.downsample = Shortcut(nn.Sequential(nn.Hardswish(inplace=True), block.downsample[0]), block.downsample[1])
    else:
        block.conv1.__class__ = Gated
    x = torch.randn(4, 3, 64, 64, device="cuda")

    def grads(net):
        with torch.autocast("cuda", dtype=torch.bfloat16):
            net(x).float().square().mean().backward()
        return [p.grad for p in net.parameters()]
    own, called = copy.deepcopy(net), copy.deepcopy(net)
    for stage in (called.layer1, called.layer2, called.layer3, called.layer4):
        stage.register_forward_hook(lambda *a: None)     # the stages are called
    for u, v in zip(grads(own), grads(called)):
        assert rel(u, v.double()) < 2e-2


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(2, 8, 3, 5), (24, 64, 56, 56)])
def test_captured_in_a_graph(shape):
    """Launches behind the previous kernel under stream capture: a replay on other values gives what the calls one by one give."""
    from aluminum_b200.ops import batch_norm_act_twice
    torch.manual_seed(0)
    cl = dict(memory_format=torch.channels_last)
    rand = lambda: torch.randn(shape, device="cuda").bfloat16().contiguous(**cl)
    bns, relu = [nn.BatchNorm2d(shape[1]).cuda() for _ in range(2)], nn.ReLU()
    start = copy.deepcopy(bns)
    x, r, dy = rand().requires_grad_(), rand().requires_grad_(), rand()

    def step(bns, x, r, dy):
        y = batch_norm_act(bns[0], x, relu)
        a, b = batch_norm_act_twice(bns[1], y + 0, relu, r)     # (behind a kernel of the framework's and behind ones of its own)
        return torch.autograd.grad([a, b], [x, r] + [p for m in bns for p in m.parameters()], [dy, dy]), a
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step(bns, x, r, dy)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        grads, y = step(bns, x, r, dy)
    for m, s in zip(bns, start):
        m.load_state_dict(s.state_dict())
    for _ in range(3):
        with torch.no_grad():
            for t in (x, r, dy):
                t.copy_(rand())
        graph.replay()
        want, z = step(start, x.detach().requires_grad_(), r.detach().requires_grad_(), dy)
        assert torch.equal(y, z) and all(torch.equal(g, w) for g, w in zip(grads, want))
        assert all(torch.equal(u, v) for m, s in zip(bns, start) for u, v in zip(m.buffers(), s.buffers()))


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(24, 64, 56), (64, 64, 112), (64, 256, 56), (96, 512, 28)])
@pytest.mark.parametrize("first", ["image", "rows"])
def test_statistics_of_rows_that_begin_far_from_the_others(shape, first):
    """A first image ten times as bright, a first stripe a thousand standard deviations off: the partial sums, and their fold, begin with them."""
    from aluminum_b200.ops import batch_norm_act
    n, c, h = shape
    torch.manual_seed(c)
    x = torch.randn(n, c, h, h, device="cuda")
    if first == "image":
        x[0] = x[0] * 10 + 10
    else:
        x[0, :, :8] += 1000
    x = x.bfloat16().contiguous(memory_format=torch.channels_last).requires_grad_()
    bn = nn.BatchNorm2d(c, momentum=1.0).cuda()
    assert "BatchNormAct" in batch_norm_act(bn, x, nn.ReLU()).grad_fn.name()
    v = x.detach().double().transpose(0, 1).flatten(1)
    mean, var = v.mean(1), v.var(1)
    # fp32 (roundings of 2^-24): a quarter of one of the standard deviation, over means of many rows, and two of the mean; eight of the variance
    assert ((bn.running_mean - mean).abs() <= 2 ** -26 * var.sqrt() + 2 ** -23 * mean.abs()).all()
    assert ((bn.running_var - var).abs() <= 2 ** -21 * var).all()
