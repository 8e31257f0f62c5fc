"""The calls on tensors in native code (src/torch/comm_calls.hpp): what they refuse, what they leave to Python, and that both agree."""
import gc

import pytest
import torch

from aluminum_b200 import _lib


@pytest.fixture(scope="module")
def calls():
    native = _lib.calls()
    if native is None:
        pytest.skip("built without Python's or PyTorch's headers")
    return native


def coll(calls, handle, ranks, send, recv, inplace=False):
    return calls.collective(handle, ranks, _lib.KINDS["allreduce"], send, recv, 1, -1, 0, 0, inplace, 1.0, 0, 0, 0, False)


class Sub(torch.Tensor):
    pass


def test_what_is_refused_and_what_is_left_to_python(calls):
    t = torch.zeros(4)
    for send, ranks, error in (([t] * 3, 2, "expected 2 tensors"), (t, 2, "takes a list"), ([t, t], 2, "contiguous CUDA tensors")):
        with pytest.raises(_lib.AlError, match=error):
            coll(calls, 0, ranks, send, send)
    for send in ([t.as_subclass(Sub)] * 2, [1, 2], [t.to(torch.complex64)] * 2, [None, None], None):
        assert coll(calls, 0, 2, send, None, False) is NotImplemented
    rows = [[1, 1]] * 2
    with pytest.raises(_lib.AlError, match="2 row"):
        calls.exchange_rows(0, 2, 2, [t] * 2, [t] * 2, 4, 4, 4, rows, rows, [[1]] * 2, rows, rows, rows, None, None, 0, False)
    with pytest.raises(_lib.AlError, match="int64"):
        calls.exchange_rows(0, 2, 2, [t] * 2, [t] * 2, 4, 4, 4, rows, rows, rows, rows, rows, rows, [t] * 2, None, 0, False)
    with pytest.raises(_lib.AlError, match="closed"):
        calls.p2p(None, 0, [(True, 1, t)], 0, False)
    with pytest.raises(TypeError):
        calls.p2p(None, 0, [(True, "x", t)], 0, False)
    assert calls.p2p(0, 0, [(True, 1)], 0, False) is NotImplemented and calls.p2p(0, 0, iter(()), 0, False) is NotImplemented


def test_tables_and_ranks_of_any_kind_are_left_to_python(calls):
    """Ranges, arrays, tensors and other numbers than ints: Python converts them."""
    import numpy as np
    t, rows = torch.zeros(4), [[1, 1]] * 2

    def call(ranks, table):
        x = [t] * ranks if ranks > 1 else t
        other = rows[:ranks]
        return calls.exchange_rows(0, ranks, 2, x, x, 4, 4, 4, other, other, table, other, other, other, None, None, 0, False)
    for table in ([range(0, 8, 4)] * 2, np.ones((2, 2), dtype=np.int64), torch.ones(2, 2, dtype=torch.int64), [np.ones(2, dtype=np.int64)] * 2,
                  [[1.0, 1.0]] * 2, [[np.int64(1)] * 2] * 2, iter([[1, 1], [1, 1]])):
        assert call(2, table) is NotImplemented
    for table in (range(0, 8, 4), np.ones(2, dtype=np.int64), torch.ones(2, dtype=torch.int64), [range(2)], (1.0, 2.0)):
        assert call(1, table) is NotImplemented
    for table in ([1, 1], (1, 1), [[1, 1]], ((True, 1),)):
        with pytest.raises(_lib.AlError, match="closed"):
            call(1, table)
    assert calls.p2p(0, 0, [(True, 1.0, t)], 0, False) is NotImplemented and calls.p2p(0, 0, [(True, 1, t, 0.0)], 0, False) is NotImplemented


def test_new_tensors(calls):
    like = [torch.zeros(1), torch.zeros(1, dtype=torch.int16)]
    for shapes, want in (((3, 4), [(3, 4)] * 2), ([(0,), (2, 5)], [(0,), (2, 5)])):
        made = calls.empties(like, shapes)
        assert [tuple(m.shape) for m in made] == want and [m.dtype for m in made] == [torch.float32, torch.int16]
    assert calls.empties([1], (2,)) is NotImplemented
    with pytest.raises(_lib.AlError):
        calls.empties(like, [(1,)])
    with pytest.raises(RuntimeError):
        calls.empties(like, (-1,))


@pytest.mark.gpu
@pytest.mark.parametrize("p", [2, 8])
def test_python_and_native_calls_agree(p):
    import aluminum_b200 as al
    from aluminum_b200.parallel import context, expert, ulysses
    al.init()
    comm = al.DeviceComm(emulate=p)
    native = comm._calls
    assert native is not None

    def everything():
        g = torch.Generator(device="cuda").manual_seed(1)
        rand = lambda *s, d=torch.float32: [torch.randint(-8, 8, s, generator=g, device="cuda").to(d) for _ in range(p)]
        out = []
        for n, d in ((5, torch.float32), (1000, torch.bfloat16), (700_000, torch.float32), (3000, torch.int32)):
            x, y = rand(n * p, d=d), rand(n * p, d=d)
            comm.allreduce(x, tuple(y))
            comm.allreduce(x, op="max")
            r = rand(n, d=d)
            comm.reduce_scatter(y, r)
            comm.allgather(r, x)
            out += x + y + r
        x = rand(9000)
        req = comm.allreduce(x, scale=0.25, wire_dtype=torch.bfloat16, nonblocking=True, stream=None)
        req.wait()
        half = [torch.empty(9000, device="cuda", dtype=torch.float16) for _ in range(p)]
        comm.allreduce(x, half, algo="one_shot")
        comm.bcast(x, root=p - 1)
        out += x + half
        u = rand(24, 2 * p, 16, d=torch.bfloat16)
        h = ulysses.seq_to_head(comm, u)
        out += h + ulysses.head_to_seq(comm, h)
        toks = rand(50, 24)
        dest = [torch.randint(0, p, (50,), generator=g, device="cuda") for _ in range(p)]
        got, state = expert.dispatch(comm, toks, dest)
        out += got + expert.combine(comm, got, state)
        ring = [torch.empty_like(t) for t in toks]
        context.ring_pass(comm, toks, ring, nonblocking=True).wait()
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        comm.allreduce(ring, stream=s)
        torch.cuda.current_stream().wait_stream(s)
        return [o.clone() for o in out + ring]
    want = everything()
    comm._calls = None
    try:
        got = everything()
    finally:
        comm._calls = native
    assert len(want) == len(got) and all(torch.equal(a, b) for a, b in zip(want, got))
    # an operation under way keeps its tensors, whatever becomes of the caller's list
    xs = [torch.ones(1 << 20, device="cuda") for _ in range(p)]
    addresses = [x.data_ptr() for x in xs]
    req = comm.allreduce(xs, nonblocking=True)
    xs.clear()
    gc.collect()
    assert [t.data_ptr() for t in req._keep[1]] == addresses
    req.wait()
    with pytest.raises(KeyError):
        comm.allreduce([torch.ones(4, device="cuda")] * p, op="nothing")
    comm.close()
    with pytest.raises(al.AlError, match="closed"):
        comm.allreduce([torch.ones(4, device="cuda") for _ in range(p)])


class Same(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        return x.clone()

    @staticmethod
    def backward(ctx, g):
        return g


def test_gradients_are_lent_where_nothing_looks_at_them(calls):
    nn, keep = torch.nn, []

    def node_hook(net):
        keep.append(net[0].weight.expand_as(net[0].weight).grad_fn.next_functions[0][0])
        keep[-1].register_hook(lambda *a: None)

    def lent(hook=None, use=lambda x: x, own=True):
        net = nn.Sequential(nn.Linear(3, 4), nn.Linear(4, 2))
        params = list(net.parameters())
        for p in params:
            p.grad = torch.zeros_like(p)
        views = [p.grad for p in params]
        if hook is not None:
            hook(net)
        if not own:
            params[1].grad = None
        was = [p.grad for p in params]
        loss = use(net(torch.randn(5, 3))).sum()
        if not calls.lend_gradients(loss, params, views):
            assert all(p.grad is g for p, g in zip(params, was))
            return False
        assert all(p.grad is None for p in params)
        loss.backward()
        calls.return_gradients(params, views)
        assert all(p.grad is v and v.any() for p, v in zip(params, views))
        return True
    assert lent() and lent(use=lambda x: x.relu().double()) and not lent(own=False)
    for hook in (lambda n: n[0].weight.register_hook(lambda g: None), lambda n: n[0].weight.register_post_accumulate_grad_hook(lambda p: None),
                 lambda n: n[1].register_full_backward_hook(lambda *a: None), lambda n: n[1].register_full_backward_pre_hook(lambda *a: None),
                 lambda n: n[0].register_forward_hook(lambda m, i, o: o.register_hook(lambda g: None) and None), node_hook,
                 lambda n: torch.autograd.graph.register_multi_grad_hook(list(n.parameters()), lambda *a: None)):
        assert not lent(hook)

    def long(x):
        for k in range(3000):      # (more nodes than the walk's first table holds, met more than once)
            x = x + x * 1e-6 if k % 100 == 0 else x + 0
        return x
    assert lent(use=long) and not lent(lambda n: n[0].weight.register_hook(lambda g: None), long)
    assert not lent(use=Same.apply) and not calls.lend_gradients(None, [], []) and not calls.lend_gradients(torch.zeros(1), [], [])
