"""The copying, converting and folding loops of the staged kernels where they can go wrong: lengths around a 16-byte word,
a warp's round and a CTA's share, buffers and slices at any byte offset, and what a rank contributes to its own
result (which skips the staging area), in place and out of place."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def al():
    import aluminum_b200 as al
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    al.init()
    yield al


@pytest.fixture(scope="module", params=[2, 3, 4, 8])
def comm(al, request):
    c = al.DeviceComm(emulate=request.param)
    yield c
    c.close()


def small_ints(n, dtype, seed, shift=0):
    """n integers of a few bits (sums are exact in every type), `shift` elements into their allocation."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(-6, 7, (n + shift,), generator=g, device="cuda").to(dtype)[shift:]


SIZES = [1, 3, 8, 129, 4099, 32768 + 5, 300001]


@pytest.mark.parametrize("dtype", [torch.uint8, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shift", [0, 1, 3])
def test_moves_at_any_offset(comm, dtype, shift):
    p = comm.size
    for n in SIZES:
        xs = [small_ints(n, dtype, r, shift) for r in range(p)]
        outs = [small_ints(p * n, dtype, 99, shift) for _ in range(p)]
        comm.allgather(xs, outs, algo="staged")
        for o in outs:
            assert torch.equal(o, torch.cat(xs))
        full = [small_ints(p * n, dtype, 50 + r, shift) for r in range(p)]
        comm.alltoall(full, outs, algo="staged")
        for r in range(p):
            assert torch.equal(outs[r], torch.cat([f[r * n:(r + 1) * n] for f in full]))
        # in place: the own slice stays where it is
        want = torch.cat([full[r][r * n:(r + 1) * n] for r in range(p)])
        both = [f.clone() for f in full]
        comm.allgather(both, algo="staged")
        for b in both:
            assert torch.equal(b, want)
        both = [f.clone() for f in full]
        comm.alltoall(both, algo="staged")
        for r in range(p):
            assert torch.equal(both[r], torch.cat([f[r * n:(r + 1) * n] for f in full]))


@pytest.mark.parametrize("dtype", [torch.int32, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shift", [0, 1])
def test_reductions_at_any_offset(comm, dtype, shift):
    p = comm.size
    for n in SIZES:
        for algo in ("one_shot", "two_shot"):
            xs = [small_ints(n, dtype, r, shift) for r in range(p)]
            want = sum(x.float() for x in xs).to(dtype)
            outs = [small_ints(n, dtype, 99, shift) for _ in range(p)]
            comm.allreduce(xs, outs, algo=algo)
            for o in outs:
                assert torch.equal(o, want)
            comm.allreduce(xs, algo=algo)
            for x in xs:
                assert torch.equal(x, want)
        full = [small_ints(p * n, dtype, 50 + r, shift) for r in range(p)]
        want = sum(f.float() for f in full).to(dtype)
        outs = [small_ints(n, dtype, 99, shift) for _ in range(p)]
        comm.reduce_scatter(full, outs, algo="staged")
        for r in range(p):
            assert torch.equal(outs[r], want[r * n:(r + 1) * n])
        comm.reduce_scatter(full, algo="staged")
        for r in range(p):
            assert torch.equal(full[r][:n], want[r * n:(r + 1) * n])


def test_partly_overlapping_buffers_stay_staged(comm):
    """A receive buffer that begins inside the send buffer: the whole input is read before anything is written."""
    p, n = comm.size, 4096 + 3
    bufs = [small_ints(3 * p * n, torch.float32, r) for r in range(p)]
    send, recv = [b[:p * n] for b in bufs], [b[n // 2:n // 2 + p * n] for b in bufs]
    want = [torch.cat([s[r * n:(r + 1) * n] for s in send]) for r in range(p)]
    comm.alltoall(send, recv, algo="staged")
    for r in range(p):
        assert torch.equal(recv[r], want[r])


@pytest.mark.parametrize("wire", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shift", [0, 1])
def test_converted_wire(comm, wire, shift):
    p = comm.size
    for n in SIZES:
        for algo in ("one_shot", "two_shot"):
            xs = [small_ints(n, torch.float32, r, shift) for r in range(p)]
            want = sum(xs)
            comm.allreduce(xs, wire_dtype=wire, algo=algo)
            for x in xs:
                assert torch.equal(x, want)   # integers of at most 48: exact in both 16-bit types

