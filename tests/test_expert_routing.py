"""Which inputs a token dispatch refuses, before anything is launched."""
from types import SimpleNamespace

import pytest
import torch

from aluminum_b200 import _lib
from aluminum_b200.parallel import expert


def test_host_memory_never_reaches_the_kernel(monkeypatch):
    """The routing kernel reads and writes plain addresses: destinations that are not on the communicator's GPU, or not one
    tensor per rank, raise before the library is called."""
    called = []
    monkeypatch.setattr(_lib, "load", lambda: called.append(1) or pytest.fail("the library was called"))
    comm = SimpleNamespace(size=2, nlocal=2, device_index=0, _h=None, _stream=lambda: None)
    dest = torch.tensor([0, 1, 1])
    for dests in ([dest, dest], [dest], [dest] * 3):
        with pytest.raises(_lib.AlError):
            expert._route(comm, dests)
        with pytest.raises(_lib.AlError):
            expert.dispatch(comm, [torch.zeros(3, 4)] * len(dests), dests)
    assert not called


@pytest.mark.gpu
def test_refused_inputs_leave_the_communicator_usable():
    import aluminum_b200 as al
    al.init()
    comm = al.DeviceComm(emulate=2)
    toks = [torch.arange(12., device="cuda").view(3, 4) + r for r in range(2)]
    dest = torch.tensor([1, 0, 1], device="cuda")
    for bad_toks, bad, error in ((toks, [dest, dest.cpu()], _lib.AlError), (toks, [dest.cpu(), dest.cpu()], _lib.AlError),
                                 (toks, [dest], _lib.AlError), ([toks[0], toks[1].cpu()], [dest, dest], _lib.AlError),
                                 (toks, [dest, dest.repeat(2)], ValueError), (toks, [dest, dest.bool()], ValueError),
                                 (toks, [dest, dest.float()], ValueError), (toks, [dest, dest.view(3, 1)], ValueError)):
        with pytest.raises(error):
            expert.dispatch(comm, bad_toks, bad)
    got, state = expert.dispatch(comm, toks, [dest, dest.to(torch.uint8)])
    assert torch.equal(got[0], torch.stack([toks[0][1], toks[1][1]]))
    back = expert.combine(comm, got, state)
    assert all(torch.equal(b, t) for b, t in zip(back, toks))
    comm.close()


@pytest.mark.parametrize("p", [1, 2, 8])
@pytest.mark.parametrize("n", [0, 1, 33, 5000])
def test_order_and_counts_by_sorting(p, n):
    d = torch.randint(0, p, (n,), generator=torch.Generator().manual_seed(n))
    counts = torch.empty(p, dtype=torch.int64)
    assert torch.equal(expert._sorted_route(d, p, counts), torch.argsort(d, stable=True))
    assert torch.equal(counts, torch.bincount(d, minlength=p))
    for wrong in (-1, p) if n else ():
        bad = d.clone()
        bad[n // 2] = wrong
        expert._sorted_route(bad, p, counts)
        assert (counts == -1).all()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [410_000, 410_001])
def test_either_side_of_the_sorting_limit(n):
    import aluminum_b200 as al
    al.init()
    comm = al.DeviceComm(emulate=2)
    dests = [torch.randint(0, 2, (n,), device="cuda"), torch.randint(0, 2, (5,), device="cuda")]
    order, both = expert._route(comm, dests)
    for r in range(2):
        assert torch.equal(order[r], torch.argsort(dests[r], stable=True))
        assert torch.equal(both[0][r], torch.bincount(dests[r], minlength=2))
    comm.close()


@pytest.mark.gpu
@pytest.mark.parametrize("p", [2, 8])
@pytest.mark.parametrize("tokens", [1, 31, 255, 256, 257, 8191, 8193, 30000])
def test_counts_that_the_host_polls(p, tokens):
    """Around what a warp keeps in registers (8 rows of 32 tokens, 32 warps); several calls, also from threads at once; refused under capture."""
    import threading
    import aluminum_b200 as al
    al.init()
    comm = al.DeviceComm(emulate=p)
    g = torch.Generator(device="cuda").manual_seed(tokens)
    dests = [[torch.randint(0, p, (max(0, tokens - r),), generator=g, device="cuda") for r in range(p)] for _ in range(6)]

    def one(d):
        order, counts = expert._route(comm, d, read=True)
        for r in range(p):
            assert counts[r] == torch.bincount(d[r], minlength=p).tolist()
            assert torch.equal(order[r], torch.argsort(d[r], stable=True))
    for d in dests:
        one(d)
    failed = []

    def run(d):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                one(d)
        except BaseException as e:
            failed.append(e)
    torch.cuda.synchronize()
    threads = [threading.Thread(target=run, args=(d,)) for d in dests]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not failed, failed
    bad = [d.clone() for d in dests[0]]
    bad[0][-1] = p
    assert expert._route(comm, bad, read=True)[1][0] == [-1] * p
    s = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with pytest.raises(_lib.AlError, match="captured"):
        with torch.cuda.graph(graph, stream=s):
            expert._route(comm, dests[0], read=True)
    one(dests[1])
    comm.close()
