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


@pytest.mark.parametrize("p", [2, 3, 4, 8])
@pytest.mark.parametrize("stage", [1 << 20, 64 << 20])
def test_large_operations_in_bulk_copies(al, p, stage):
    """Around tiles of 32 KiB, shares of a CTA and (small staging) several chunks; ragged vectors, in place and not."""
    old = al.get_tuning("dev_stage_bytes")
    al.set_tuning("dev_stage_bytes", stage)
    comm = al.DeviceComm(emulate=p)
    al.set_tuning("dev_stage_bytes", old)
    for dtype, n in ((torch.float32, 262144), (torch.float32, 1310727), (torch.bfloat16, 524288 + 9), (torch.bfloat16, 3000003)):
        xs = [small_ints(n, dtype, r) for r in range(p)]
        want = sum(x.float() for x in xs).to(dtype)
        outs = [torch.empty_like(x) for x in xs]
        comm.allreduce(xs, outs, algo="two_shot" if p > 2 else "auto")
        assert all(torch.equal(o, want) for o in outs)
        comm.allreduce(xs, algo="two_shot" if p > 2 else "one_shot")
        assert all(torch.equal(x, want) for x in xs)
    for wire, n in ((torch.bfloat16, 524288), (torch.float16, 1310727), (torch.bfloat16, 3000003)):
        xs = [small_ints(n, torch.float32, r) for r in range(p)]
        want = sum(xs)
        outs = [torch.empty_like(x) for x in xs]
        comm.allreduce(xs, outs, wire_dtype=wire)
        assert all(torch.equal(o, want) for o in outs)
        comm.allreduce(xs, wire_dtype=wire)
        assert all(torch.equal(x, want) for x in xs)
    for dtype, n in ((torch.bfloat16, 262144), (torch.float32, 131072 * 3 + 4), (torch.float32, 655360 + 12),
                     (torch.bfloat16, 524288 + 1), (torch.float32, 262144 + 3), (torch.bfloat16, 1310720 + 13)):
        full = [small_ints(p * n, dtype, 50 + r) for r in range(p)]
        want = sum(f.float() for f in full).to(dtype)
        outs = [torch.empty(n, device="cuda", dtype=dtype) for _ in range(p)]
        comm.reduce_scatter(full, outs, algo="staged")
        assert all(torch.equal(outs[r], want[r * n:(r + 1) * n]) for r in range(p))
        all_outs = [torch.empty_like(f) for f in full]
        comm.allgather(outs, all_outs, algo="staged")
        assert all(torch.equal(o, want) for o in all_outs)
        comm.alltoall(full, all_outs, algo="staged")
        moved = [torch.cat([f[r * n:(r + 1) * n] for f in full]) for r in range(p)]
        assert all(torch.equal(all_outs[r], moved[r]) for r in range(p))
        both = [f.clone() for f in full]
        comm.alltoall(both, algo="staged")
        assert all(torch.equal(both[r], moved[r]) for r in range(p))
        both = [f.clone() for f in full]
        comm.reduce_scatter(both, algo="staged")
        assert all(torch.equal(both[r][:n], want[r * n:(r + 1) * n]) for r in range(p))
        both = [f.clone() for f in full]
        comm.allgather(both, algo="staged")
        assert all(torch.equal(b, torch.cat([full[r][r * n:(r + 1) * n] for r in range(p)])) for b in both)
    comm.close()


@pytest.mark.parametrize("p", [2, 4, 8])
@pytest.mark.parametrize("width,rows", [(16, 1), (16, 1000), (80, 333), (1024, 67), (4096, 5), (4112, 31), (12000, 9), (24, 77), (7, 50)])
def test_rows_of_any_length(al, p, width, rows):
    """Rows of `width` bytes: several to a warp's round, one, more than one round, and lengths that are no whole words."""
    comm = al.DeviceComm(emulate=p)
    table = lambda v: [v] * p
    x = [small_ints(p * rows * width, torch.uint8, r).view(rows, p, width) for r in range(p)]
    order = [torch.randperm(rows, generator=torch.Generator().manual_seed(r)).cuda() for r in range(p)]
    out = [torch.zeros(p, rows, width, device="cuda", dtype=torch.uint8) for _ in range(p)]
    comm.exchange_rows(x, out, width, p * width, width, table([rows] * p), table([0] * p), table([d * width for d in range(p)]),
                       table([rows] * p), table([s * rows for s in range(p)]), table([0] * p), send_idx=order)
    for r in range(p):
        for s in range(p):
            assert torch.equal(out[r][s], x[s][order[s], r])
    comm.close()


@pytest.mark.parametrize("p", [2, 3, 8])
@pytest.mark.parametrize("tokens", [0, 1, 31, 32, 33, 1024, 1025, 40000])
def test_routing_order_and_counts(al, p, tokens):
    from aluminum_b200.parallel import expert
    comm = al.DeviceComm(emulate=p)
    g = torch.Generator(device="cuda").manual_seed(tokens)
    dests = [torch.randint(0, p, (tokens,), generator=g, device="cuda") // (1 + r % 2) for r in range(p)]
    order, both = expert._route(comm, dests)
    for r in range(p):
        assert torch.equal(order[r], torch.argsort(dests[r], stable=True))
        assert torch.equal(both[0][r], torch.bincount(dests[r], minlength=p))
    if tokens:
        toks = [torch.zeros(tokens, 8, device="cuda") for _ in range(p)]
        for wrong in (-1, p):
            bad = [d.clone() for d in dests]
            bad[0][-1] = wrong
            with pytest.raises(ValueError):
                expert.dispatch(comm, toks, bad)
    comm.close()


@pytest.mark.parametrize("n", [4099, 262144])   # (262144 fp32: where the bulk copy engine takes over; one chunk)
def test_receive_buffers_that_are_other_ranks_send_buffers(comm, n):
    """With all ranks in one process a rank's result may land on what another rank still has to send: everything is read first."""
    p = comm.size
    fresh = lambda m: [small_ints(m, torch.float32, r) for r in range(p)]
    turn = lambda bufs: bufs[1:] + bufs[:1]      # rank r receives where rank r + 1 sends from
    for algo in ("one_shot", "two_shot"):
        xs = fresh(n)
        want = sum(xs)
        comm.allreduce(xs, turn(xs), algo=algo)
        assert all(torch.equal(x, want) for x in xs)
    full = fresh(p * n)
    want = [f.clone() for f in full]
    comm.alltoall(full, turn(full), algo="staged")
    for r, got in enumerate(turn(full)):
        assert torch.equal(got, torch.cat([f[r * n:(r + 1) * n] for f in want]))
    full = fresh(p * n)
    want = sum(full)
    place = lambda r: slice((r + 1) % p * n, ((r + 1) % p + 1) * n)   # the slice that rank r + 1 contributes to its own result
    comm.reduce_scatter(full, [f[place(r)] for r, f in enumerate(turn(full))], algo="staged")
    for r, f in enumerate(turn(full)):
        assert torch.equal(f[place(r)], want[r * n:(r + 1) * n])
    full = fresh(p * n)
    shards = [f[:n] for f in full]
    want = torch.cat([s.clone() for s in shards])
    comm.allgather(shards, turn(full), algo="staged")
    assert all(torch.equal(f, want) for f in full)


@pytest.mark.parametrize("threads", [16, 100, 333, 511])
def test_threads_that_are_no_whole_warps(al, comm, threads):
    """The loops deal in rounds of a warp; a tuning that is no multiple of one is rounded, not half obeyed."""
    p, old = comm.size, al.get_tuning("threads_per_cta")
    al.set_tuning("threads_per_cta", threads)
    try:
        for n in (4099, 300001):
            for dtype, algo in ((torch.float32, "one_shot"), (torch.float32, "two_shot"), (torch.int32, "one_shot")):
                xs = [small_ints(n, dtype, r) for r in range(p)]
                want = sum(xs)
                outs = [torch.zeros_like(x) for x in xs]
                comm.allreduce(xs, outs, algo=algo)
                assert all(torch.equal(o, want) for o in outs)
            xs = [small_ints(n, torch.uint8, r) for r in range(p)]
            outs = [torch.zeros(p * n, device="cuda", dtype=torch.uint8) for _ in range(p)]
            comm.allgather(xs, outs, algo="staged")
            assert all(torch.equal(o, torch.cat(xs)) for o in outs)
    finally:
        al.set_tuning("threads_per_cta", old)


def bulk_from(p, wire=False):
    """Bytes of a vector from which the bulk copies take an operation of p ranks."""
    return (16 if p == 2 else (32 if wire else 8) if p <= 4 else (2 if wire else 1)) << 20


@pytest.mark.parametrize("limits", [dict(max_ctas=1, max_ctas_pipelined=2), dict(max_ctas=5, max_ctas_pipelined=3), dict(threads_per_cta=256)])
def test_bulk_copies_within_the_callers_limits(al, comm, limits):
    """Grid sizes down to one CTA per rank (many rounds of tiles each), and smaller CTAs, for which the loops stand in."""
    p, old = comm.size, {k: al.get_tuning(k) for k in limits}
    for k, v in limits.items():
        al.set_tuning(k, v)
    try:
        for n in (bulk_from(p) // 4 + 9, bulk_from(p, True) // 4 + 900003):
            xs = [small_ints(n, torch.float32, r) for r in range(p)]
            want = sum(xs)
            outs = [torch.empty_like(x) for x in xs]
            comm.allreduce(xs, outs, algo="two_shot")
            assert all(torch.equal(o, want) for o in outs)
            comm.allreduce(xs, wire_dtype=torch.bfloat16)
            assert all(torch.equal(x, want) for x in xs)
        n = 2097152 + 5
        full = [small_ints(p * n, torch.float32, r) for r in range(p)]
        want = sum(full)
        outs = [torch.empty(n, device="cuda") for _ in range(p)]
        comm.reduce_scatter(full, outs, algo="staged")
        assert all(torch.equal(outs[r], want[r * n:(r + 1) * n]) for r in range(p))
        both = [torch.empty_like(f) for f in full]
        comm.allgather(outs, both, algo="staged")
        assert all(torch.equal(b, want) for b in both)
    finally:
        for k, v in old.items():
            al.set_tuning(k, v)


def test_which_operations_the_bulk_copies_take(al, comm):
    p = comm.size

    def taken(call):
        before = comm.stats()["bulk_staged"]
        call()
        return comm.stats()["bulk_staged"] - before
    n = bulk_from(p, True) // 4 + 12
    xs = [small_ints(n, torch.float32, r) for r in range(p)]
    want = sum(xs)
    outs = [torch.empty_like(x) for x in xs]
    for wire in (None, torch.bfloat16):
        least = bulk_from(p, wire is not None) // 4
        for algo in ("one_shot", "two_shot"):
            for m in (least, least + 9, n):
                assert taken(lambda: comm.allreduce([x[:m] for x in xs], [o[:m] for o in outs], wire_dtype=wire, algo=algo)) == 1
                assert all(torch.equal(o[:m], want[:m]) for o in outs)
            assert taken(lambda: comm.allreduce([x[:least - 4] for x in xs], [o[:least - 4] for o in outs], wire_dtype=wire, algo=algo)) == 0
    # nor: operators other than sums, a grid size of the caller's own, smaller CTAs, unaligned buffers
    assert taken(lambda: comm.allreduce(xs, outs, "max", algo="one_shot")) == 0
    assert taken(lambda: comm.allreduce(xs, outs, algo="one_shot", ctas=4)) == 0
    shifted = [small_ints(n, torch.float32, r, 1) for r in range(p)]
    assert taken(lambda: comm.allreduce(shifted, outs, algo="one_shot")) == 0
    assert all(torch.equal(o, sum(shifted)) for o in outs)
    old = al.get_tuning("threads_per_cta")
    al.set_tuning("threads_per_cta", 256)
    assert taken(lambda: comm.allreduce(xs, outs, algo="one_shot")) == 0
    al.set_tuning("threads_per_cta", old)


@pytest.mark.parametrize("stage", [1 << 20, 64 << 20])
@pytest.mark.parametrize("dtype,odd", [(torch.float32, 0), (torch.bfloat16, 7), (torch.float16, 8)])
def test_bulk_copies_from_their_smallest_sizes_on(al, stage, dtype, odd):
    """Reductions where the bulk copies begin, in one chunk and (small staging) in many."""
    old = al.get_tuning("dev_stage_bytes")
    al.set_tuning("dev_stage_bytes", stage)
    for p in (2, 3, 4):
        comm = al.DeviceComm(emulate=p)
        n = bulk_from(p) // dtype.itemsize + odd
        xs = [small_ints(n, dtype, r) for r in range(p)]
        want = sum(x.float() for x in xs).to(dtype)
        outs = [torch.empty_like(x) for x in xs]
        for algo in ("one_shot", "two_shot"):
            comm.allreduce(xs, outs, algo=algo)
            assert all(torch.equal(o, want) for o in outs)
        m = bulk_from(p) // dtype.itemsize // p // 8 * 8 + 8 + odd
        full = [small_ints(p * m, dtype, 9 + r) for r in range(p)]
        want = sum(f.float() for f in full).to(dtype)
        outs = [torch.empty(m, device="cuda", dtype=dtype) for _ in range(p)]
        comm.reduce_scatter(full, outs, algo="staged")
        assert all(torch.equal(o, want[r * m:(r + 1) * m]) for r, o in enumerate(outs))
        assert comm.stats()["bulk_staged"] == 3
        comm.close()
    al.set_tuning("dev_stage_bytes", old)


@pytest.mark.parametrize("n", [(8 << 20) // 4, (8 << 20) // 4 + 3])   # 16 MiB in all on two ranks: where their bulk copies begin
def test_large_moves(al, comm, n):
    p = comm.size
    full = [small_ints(p * n, torch.int32, r) for r in range(p)]
    outs = [torch.empty_like(f) for f in full]
    before = comm.stats()["bulk_staged"]
    comm.alltoall(full, outs, algo="staged")
    assert all(torch.equal(outs[r], torch.cat([f[r * n:(r + 1) * n] for f in full])) for r in range(p))
    shards = [f[:n] for f in full]
    comm.allgather(shards, outs, algo="staged")
    assert all(torch.equal(o, torch.cat(shards)) for o in outs)
    assert comm.stats()["bulk_staged"] == before + 2
    if p == 2:
        small = [f[:2 * n - 16] for f in full]
        comm.alltoall(small, [o[:2 * n - 16] for o in outs], algo="staged")
        assert comm.stats()["bulk_staged"] == before + 2


@pytest.mark.parametrize("shift", [64, 4096 + 4])
def test_large_partly_overlapping_buffers(al, comm, shift):
    """Where the bulk copies begin: only forms that send everything through staging may use bulk copies then (one chunk each here)."""
    p = comm.size
    n = bulk_from(p) // 4 + 4

    def buffers(m):
        base = [small_ints(m + shift, torch.float32, r) for r in range(p)]
        return [b[:m] for b in base], [b[shift:] for b in base]
    before = comm.stats()["bulk_staged"]
    for algo in ("one_shot", "two_shot"):
        xs, outs = buffers(n)
        want = sum(xs)
        comm.allreduce(xs, outs, algo=algo)
        assert all(torch.equal(o, want) for o in outs)
    m = n // p // 4 * 4     # (one chunk)
    full, outs = buffers(p * m)
    want = [torch.cat([f[r * m:(r + 1) * m] for f in full]) for r in range(p)]
    comm.alltoall(full, outs, algo="staged")
    assert all(torch.equal(o, w) for o, w in zip(outs, want))
    assert comm.stats()["bulk_staged"] == before
    for algo in ("one_shot", "two_shot"):
        xs, outs = buffers(bulk_from(p, True) // 4)
        want = sum(xs)
        comm.allreduce(xs, outs, wire_dtype=torch.bfloat16, algo=algo)
        assert all(torch.equal(o, want) for o in outs)
    m += 1   # slices that are no whole 16-byte words
    full, _ = buffers(p * m)
    want = sum(full)
    outs = [f[shift + r * m // 4 * 4:][:m] for r, f in enumerate(full)]
    comm.reduce_scatter(full, [o if o.numel() == m else f[:m] for o, f in zip(outs, full)], algo="staged")
    for r, (o, f) in enumerate(zip(outs, full)):
        assert torch.equal(o if o.numel() == m else f[:m], want[r * m:(r + 1) * m])
    assert comm.stats()["bulk_staged"] == before + 3


@pytest.mark.parametrize("p,width,rows", [(2, 2064, 33), (4, 3072, 65), (3, 4080, 7), (8, 2050, 20), (2, 4095, 40), (2, 4112, 8200), (2, 4099, 8200)])
def test_rows_in_rounds_of_four_and_eight(al, p, width, rows):
    """Rows between 2 and 4 KiB (one round of eight loads), and longer ones in an exchange of more than 128 MiB (rounds of four)."""
    comm = al.DeviceComm(emulate=p)
    table = lambda v: [v] * p
    x = [small_ints(p * rows * width, torch.uint8, r).view(p, rows, width) for r in range(p)]
    order = [torch.randperm(rows, generator=torch.Generator().manual_seed(r)).cuda() for r in range(p)]
    out = [torch.zeros(p, rows, width, device="cuda", dtype=torch.uint8) for _ in range(p)]
    offsets = table([d * rows * width for d in range(p)])
    comm.exchange_rows(x, out, width, width, width, table([rows] * p), table([0] * p), offsets, table([rows] * p), table([0] * p), offsets,
                       send_idx=order)
    for r in range(p):
        for s in range(p):
            assert torch.equal(out[r][s], x[s][r][order[s]])
    comm.close()
