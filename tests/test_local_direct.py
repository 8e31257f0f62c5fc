"""Operations of ranks that all live on one GPU, straight between their buffers (kernels/local_*.cu): every form that they
accept gives bit for bit what the staging protocol gives, and what they must not take goes through staging.

The kernels that ranks on GPUs of their own run are tested on one GPU in the other files where a call names its path or (the fixture
``local_direct``) runs both ways; the other tests there that leave it open are run again here with ``local_direct`` off.
"""
import random

import pytest
import torch

import test_device_copy_edges
import test_device_emulated
import test_device_paths

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def al():
    import aluminum_b200 as al
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    al.init()
    return al


@pytest.fixture
def staged(al):
    al.set_tuning("local_direct", 0)
    yield
    al.set_tuning("local_direct", 1)


def values(n, dtype, seed, shift=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    if not dtype.is_floating_point:
        return torch.randint(-1000, 1000, (n + shift,), generator=g, device="cuda").to(dtype)[shift:]
    return (torch.rand(n + shift, generator=g, device="cuda", dtype=torch.float64) * 2 - 1).to(dtype)[shift:]


def both(al, comm, call, taken=1):
    """The results of call() straight between buffers and through staging; `taken`: how many operations the first way took."""
    before = comm.stats()["local"]
    direct = call()
    assert comm.stats()["local"] - before == taken
    al.set_tuning("local_direct", 0)
    try:
        old = call()
    finally:
        al.set_tuning("local_direct", 1)
    assert comm.stats()["local"] - before == taken
    torch.cuda.synchronize()
    assert comm.status()["code"] == 0
    return direct, old


def same(direct, old):
    for a, b in zip(direct, old):
        assert torch.equal(a.view(torch.uint8) if a.dtype != torch.uint8 else a, b.view(torch.uint8) if b.dtype != torch.uint8 else b)


# beyond what travels as packets (2 MiB per rank at most), around whole words and warps' shares
LENGTHS = [3 << 20, (3 << 20) + 2, (3 << 20) + 18, (5 << 20) + 1034]


@pytest.mark.parametrize("p", [2, 3, 4, 5, 8])
@pytest.mark.parametrize("dtype,ops", [(torch.float32, ("sum", "avg", "min", "max")), (torch.bfloat16, ("sum", "max")), (torch.float16, ("avg", "min")),
                                       (torch.float64, ("sum", "max")), (torch.int32, ("sum", "avg", "min")), (torch.int64, ("sum", "max"))])
def test_allreduce_equals_staging(al, p, dtype, ops):
    comm = al.DeviceComm(emulate=p)
    for k, nbytes in enumerate(LENGTHS):
        n = nbytes // dtype.itemsize
        op = ops[k % len(ops)]
        for shift, out_shift in ((0, 0), (1, 0), (0, 1), (1, 1)):
            def out_of_place():
                xs = [values(n, dtype, r, shift) for r in range(p)]
                whole = [torch.zeros(n + out_shift + 3, dtype=dtype, device="cuda") for _ in range(p)]
                comm.allreduce(xs, [w[out_shift:out_shift + n] for w in whole], op)
                return whole                     # with what lies before and behind the result
            same(*both(al, comm, out_of_place))

            def in_place():
                xs = [values(n, dtype, r, shift) for r in range(p)]
                comm.allreduce(xs, op=op, scale=0.375 if dtype.is_floating_point else 1.0)
                return xs
            same(*both(al, comm, in_place))
    comm.close()


@pytest.mark.parametrize("p", [2, 3, 4, 8])
@pytest.mark.parametrize("wire", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n", [1, 5, 4097, 300001, 3000009])
def test_narrower_type_between_ranks_rounds_as_staging_does(al, p, wire, n):
    comm = al.DeviceComm(emulate=p)
    for shift in (0, 1):
        def call():
            xs = [values(n, torch.float32, r, shift) for r in range(p)]
            comm.allreduce(xs, scale=1.0 / p, wire_dtype=wire)
            outs = [torch.zeros(n, device="cuda") for _ in range(p)]
            comm.allreduce(xs, outs, wire_dtype=wire)
            return xs + outs
        same(*both(al, comm, call, 2))
    comm.close()


@pytest.mark.parametrize("p", [2, 3, 4, 8])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.int64])
def test_reduce_scatter_allgather_alltoall_equal_staging(al, p, dtype):
    comm = al.DeviceComm(emulate=p)
    for nbytes in ((2 << 20) + 16, (2 << 20) + 8 + 2 * dtype.itemsize, (3 << 20) + 5 * dtype.itemsize):
        n = nbytes // dtype.itemsize             # per slice: more than the packets carry, whole words and not
        for shift in (0, 1):
            def reduce_scatter():
                xs = [values(p * n, dtype, r, shift) for r in range(p)]
                whole = [torch.zeros(n + 3, dtype=dtype, device="cuda") for _ in range(p)]
                comm.reduce_scatter(xs, [w[:n] for w in whole])
                mine = [x[r * n:(r + 1) * n] for r, x in enumerate(xs)]   # each result on the own contribution
                comm.reduce_scatter(xs, mine)
                return whole + xs
            same(*both(al, comm, reduce_scatter, 2))

            def allgather():
                whole = [torch.zeros(p * n + 5, dtype=dtype, device="cuda") for _ in range(p)]
                comm.allgather([values(n, dtype, r, shift) for r in range(p)], [w[2 * shift:2 * shift + p * n] for w in whole])
                own = [torch.zeros(p * n + 5, dtype=dtype, device="cuda") for _ in range(p)]
                for r in range(p):
                    own[r][shift + r * n:shift + (r + 1) * n] = values(n, dtype, r)
                comm.allgather([w[shift:shift + p * n] for w in own])
                uneven = [torch.zeros(p * n + 9, dtype=dtype, device="cuda") for _ in range(p)]   # receive buffers on different addresses modulo 16
                comm.allgather([values(n, dtype, r) for r in range(p)], [w[r:r + p * n] for r, w in enumerate(uneven)])
                return whole + own + uneven
            same(*both(al, comm, allgather, 3))

            def alltoall():
                whole = [torch.zeros(p * n + 5, dtype=dtype, device="cuda") for _ in range(p)]
                comm.alltoall([values(p * n, dtype, r, shift) for r in range(p)], [w[1:1 + p * n] for w in whole])
                return whole
            same(*both(al, comm, alltoall))
    comm.close()


@pytest.mark.parametrize("limits", [dict(max_ctas=1), dict(threads_per_cta=96), dict(threads_per_cta=512, max_ctas=3)])
def test_within_the_callers_limits(al, limits):
    p, n, old = 4, 1 << 20, {k: al.get_tuning(k) for k in limits}
    comm = al.DeviceComm(emulate=p)
    for k, v in limits.items():
        al.set_tuning(k, v)
    try:
        xs = [values(n + 3, torch.float32, r) for r in range(p)]
        outs = [torch.empty_like(x) for x in xs]
        comm.allreduce(xs, outs, "max")
        assert all(torch.equal(o, torch.stack(xs).amax(0)) for o in outs)
        full = [torch.empty(p * (n + 3), device="cuda") for _ in range(p)]
        comm.allgather(xs, full)
        assert all(torch.equal(f, torch.cat(xs)) for f in full)
        assert comm.stats()["local"] == 2
    finally:
        for k, v in old.items():
            al.set_tuning(k, v)
        comm.close()


@pytest.mark.parametrize("p", [2, 3, 8])
def test_fewer_ctas_than_parts(al, p):
    """One CTA per rank, where there are p * (p - 1) copies, p * p pairs of row blocks or two planes per rank."""
    from aluminum_b200.ops import HaloExchange
    old, comm = al.get_tuning("max_ctas"), al.DeviceComm(emulate=p)
    al.set_tuning("max_ctas", 1)
    try:
        for n in (5, 1024, 40_001):
            def move():
                xs = [values(p * n, torch.float32, r) for r in range(p)]
                moved, every = ([torch.zeros(p * n + 4, device="cuda") for _ in range(p)] for _ in range(2))
                comm.alltoall(xs, [m[:p * n] for m in moved])
                comm.allgather([x[:n] for x in xs], [e[r % 4:r % 4 + p * n] for r, e in enumerate(every)])
                rows = [torch.zeros(p * n, 8, device="cuda") for _ in range(p)]
                first = [[d * n for d in range(p)] for _ in range(p)]
                comm.exchange_rows([x.view(p * n, 1).expand(p * n, 8).contiguous() for x in xs], rows, 32, 32, 32, [[n] * p for _ in range(p)], first,
                                   [[0] * p for _ in range(p)], [[n] * p for _ in range(p)], first, [[0] * p for _ in range(p)])
                return moved + every + rows
            same(*both(al, comm, move, 3))
        hx = HaloExchange(comm, 2, 3, 4, 17, 19, 2, True)

        def halo():
            for r, t in enumerate(hx.tensors):
                t.copy_(values(t.numel(), torch.float32, r).view(t.shape))
            hx.exchange()
            return [t.clone() for t in hx.tensors]
        same(*both(al, comm, halo))
    finally:
        al.set_tuning("max_ctas", old)
        comm.close()


def test_what_goes_through_staging(al):
    """Buffers that meet, in-place forms that are read elsewhere, and calls that name a path or a grid."""
    p, n = 4, 1 << 20
    comm = al.DeviceComm(emulate=p)
    xs = [values(n, torch.float32, r) for r in range(p)]
    want = torch.stack(xs).amax(0)
    turned = xs[1:] + xs[:1]

    def outs():
        return [torch.empty_like(x) for x in xs]
    for kw in (dict(algo="one_shot"), dict(algo="two_shot"), dict(ctas=4)):
        o = outs()
        comm.allreduce(xs, o, "max", **kw)
        assert all(torch.equal(v, want) for v in o)
    base = [values(n + 64, torch.float32, r) for r in range(p)]
    w = torch.stack([b[:n] for b in base]).amax(0)
    o = [b[64:] for b in base]                   # partly on the own contribution
    comm.allreduce([b[:n] for b in base], o, "max")
    assert all(torch.equal(v, w) for v in o)
    saved = [x.clone() for x in xs]
    comm.alltoall(xs, turned)                    # a receive buffer that is another rank's send buffer
    m = n // p
    assert all(torch.equal(turned[r], torch.cat([s[r * m:(r + 1) * m] for s in saved])) for r in range(p))
    ys = [x.clone() for x in saved]
    comm.alltoall(ys)
    assert all(torch.equal(ys[r], torch.cat([s[r * m:(r + 1) * m] for s in saved])) for r in range(p))
    ys = [x.clone() for x in saved]
    comm.reduce_scatter(ys, op="max")            # results at the start of buffers that are still read
    assert all(torch.equal(ys[r][:m], want[r * m:(r + 1) * m]) for r in range(p))
    comm.allreduce(saved, outs(), "prod")        # no kernel for the operator
    assert comm.stats()["local"] == 0
    comm.close()


@pytest.mark.parametrize("kind", ["allreduce", "reduce_scatter", "allgather", "alltoall"])
def test_random_forms_equal_staging(al, kind):
    rng = random.Random(kind)
    for k in range(12):
        p = rng.choice([2, 3, 4, 5, 6, 7, 8])
        dtype = rng.choice([torch.float32, torch.bfloat16, torch.float16, torch.int32])
        n = rng.randint(1_100_000, 1_900_000)   # beyond the packets in every type
        shifts = [rng.choice([0, 0, 1, 2, 3, 4, 8]) for _ in range(2 * p)]
        comm = al.DeviceComm(emulate=p)

        def call():
            send = n * (p if kind in ("reduce_scatter", "alltoall") else 1)
            recv = n * (p if kind in ("allgather", "alltoall") else 1)
            xs = [values(send, dtype, r, shifts[r]) for r in range(p)]
            whole = [torch.zeros(recv + 12, dtype=dtype, device="cuda") for _ in range(p)]
            outs = [w[shifts[p + r]:shifts[p + r] + recv] for r, w in enumerate(whole)]
            getattr(comm, kind)(xs, outs)
            return whole
        phases = {s * dtype.itemsize % 16 for s in shifts[p:]}
        same(*both(al, comm, call, 0 if kind == "allreduce" and len(phases) > 1 else 1))   # (results on different addresses modulo 16)
        comm.close()


@pytest.mark.parametrize("test", [test_device_emulated.test_pipelined_schedule, test_device_paths.test_two_rank_allreduce_is_pipelined_above_threshold])
def test_staging_between_gpus(al, staged, test):
    test(al)


@pytest.mark.parametrize("p", [2, 8])
def test_staging_between_gpus_of_large_operations(al, staged, p):
    comm = al.DeviceComm(emulate=p)
    test_device_emulated.test_reduce_scatter_allgather_alltoall(comm, 131072 * 8 + 3)
    test_device_emulated.test_allreduce_f32(comm, 3000001, "auto")
    assert comm.stats()["local"] == 0
    comm.close()


@pytest.mark.parametrize("p", [2, 3, 8])
@pytest.mark.parametrize("width,most", [(16, 300), (48, 700), (496, 90), (512, 200), (528, 33), (2048, 40), (2064, 40), (4096, 300), (12304, 9), (24, 77), (7, 50), (4099, 30)])
def test_rows_equal_staging(al, p, width, most):
    """Uneven row counts (some none), strided on one side and indexed on the other, around what a warp takes at a time."""
    comm = al.DeviceComm(emulate=p)
    counts = [[(7 * s + 13 * d * s) % (most + 1) if (s + d) % 4 else 0 for d in range(p)] for s in range(p)]
    counts[0][p - 1] = most
    back = [[counts[s][d] for s in range(p)] for d in range(p)]
    first = lambda rows: [[sum(r[:i]) for i in range(p)] for r in rows]
    zero = [[0] * p for _ in range(p)]
    for indexed in ("neither", "send", "recv"):
        def call():
            g = torch.Generator().manual_seed(3)
            x = [values(max(1, sum(counts[r])) * width, torch.uint8, r).view(-1, width) for r in range(p)]
            wide = width + (16 if width % 16 == 0 else 5)     # rows further apart than they are long
            out = [torch.zeros(max(1, sum(back[r])) * wide, dtype=torch.uint8, device="cuda") for r in range(p)]
            kw = {}
            if indexed == "send":
                kw["send_idx"] = [torch.randperm(sum(c), generator=g).cuda() for c in counts]
            if indexed == "recv":
                kw["recv_idx"] = [torch.randperm(sum(c), generator=g).cuda() for c in back]
            comm.exchange_rows(x, out, width, width, wide, counts, first(counts), zero, back, first(back), zero, **kw)
            return out
        same(*both(al, comm, call))
    comm.close()


def test_rows_that_meet_go_through_staging(al):
    p, n, w = 4, 64, 32
    comm = al.DeviceComm(emulate=p)
    rows = [[n // p] * p for _ in range(p)]
    first = [[d * (n // p) for d in range(p)] for _ in range(p)]
    zero = [[0] * p for _ in range(p)]
    x = [values(n * w, torch.uint8, r).view(n, w) for r in range(p)]
    want = [torch.cat([s[r * n // p:(r + 1) * n // p] for s in x]) for r in range(p)]
    args = (w, w, w, rows, first, zero, rows, first, zero)
    comm.exchange_rows(x, x, *args)                                   # in place
    assert all(torch.equal(a, b) for a, b in zip(x, want))
    whole = values(2 * p * n * w, torch.uint8, 9).view(2 * p, n, w)   # indexed rows may lie anywhere in a tensor's memory
    sends, recvs = [whole[2 * r] for r in range(p)], [whole[2 * r + 1] for r in range(p)]
    want = [torch.cat([s[r * n // p:(r + 1) * n // p] for s in sends]) for r in range(p)]
    order = [torch.arange(n, device="cuda") for _ in range(p)]
    before = comm.stats()["local"]
    comm.exchange_rows(sends, recvs, *args, send_idx=order)
    assert all(torch.equal(a, b) for a, b in zip(recvs, want))
    assert comm.stats()["local"] == before == 0 and comm.stats()["rows"] == 2
    comm.exchange_rows(sends, recvs, *args)                           # without indexes their places are known
    assert all(torch.equal(a, b) for a, b in zip(recvs, want))
    assert comm.stats()["local"] == 1
    comm.close()


@pytest.mark.parametrize("p", [2, 4, 8])
def test_row_exchange_between_gpus(al, staged, p):
    test_device_paths.test_row_exchange_strided_indexed_and_chunked(al, p)
    for width, rows in ((16, 1000), (80, 333), (4112, 31), (7, 50)):
        test_device_copy_edges.test_rows_of_any_length(al, p, width, rows)
    for width, rows in ((2064, 33), (4080, 7), (4112, 4200)):
        test_device_copy_edges.test_rows_in_rounds_of_four_and_eight(al, p, width, rows)


def ring(p, src, dst, step=1):
    return [x for r in range(p) for x in ((True, (r + step) % p, src[r], r), (False, (r - step) % p, dst[r], r))]


@pytest.mark.parametrize("p", [2, 3, 8])
def test_p2p_with_both_ends_in_the_call(al, p):
    comm = al.DeviceComm(emulate=p)
    for k, n in enumerate((1, 15, 16, 511, 4097, 65536, 2_097_153, 9_000_001)):
        src = [values(n, torch.uint8, r, r % 4) for r in range(p)]
        whole = [torch.zeros(n + 9, dtype=torch.uint8, device="cuda") for _ in range(p)]
        before = comm.stats()["local"]
        comm.p2p(ring(p, src, [w[3:3 + n] for w in whole]))
        assert comm.stats()["local"] == before + 1
        for r, w in enumerate(whole):
            assert torch.equal(w[3:3 + n], src[(r - 1) % p]) and not w[:3].any() and not w[3 + n:].any()
    # several messages of one pair meet in order, an empty one among them; a rank may send to itself
    msgs = [values(n, torch.float32, n) for n in (1000, 0, 70000, 3)]
    got = [torch.zeros_like(m) for m in msgs]
    comm.p2p([(True, 1, m, 0) for m in msgs[:3]] + [(True, 0, msgs[3], 0)] + [(False, 0, g, 1) for g in got[:3]] + [(False, 0, got[3], 0)])
    assert all(torch.equal(g, m) for g, m in zip(got, msgs)) and comm.status()["code"] == 0
    comm.close()


def test_p2p_order_beside_the_mailbox(al):
    """Messages of which one end came in an earlier call stay in order before those that have both ends in a call."""
    comm = al.DeviceComm(emulate=2)
    comm.set_timeout_ms(3000)
    m = [torch.full((100,), float(i), device="cuda") for i in range(5)]
    g = [torch.zeros(100, device="cuda") for _ in range(5)]
    comm.p2p([(True, 1, m[0], 0)])                                        # under way in the packet ring
    comm.p2p([(True, 1, m[1], 0), (False, 0, g[0], 1)])                   # receives the first
    comm.p2p([(False, 0, g[1], 1)])
    assert comm.stats()["local"] == 0
    comm.p2p([(True, 1, m[2], 0), (False, 0, g[2], 1), (True, 1, m[3], 0)])   # the last one is received later
    comm.p2p([(False, 0, g[3], 1)])
    comm.p2p([(True, 1, m[4], 0), (False, 0, g[4], 1)])
    assert comm.stats()["local"] == 2
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(g, m)) and comm.status()["code"] == 0
    a = [torch.full((50001,), float(r), device="cuda") for r in range(2)]
    comm.p2p(ring(2, a, a))                                               # in place
    both_ways = [torch.full((6,), float(r), device="cuda") for r in range(2)]
    comm.p2p([(True, 1, both_ways[0][:4], 0), (False, 0, both_ways[0][2:], 1)])   # the receive buffer meets the send buffer
    torch.cuda.synchronize()
    assert torch.all(a[0] == 1) and torch.all(a[1] == 0)
    assert comm.stats()["local"] == 2 and comm.status()["code"] == 0
    comm.close()


@pytest.mark.parametrize("p", [2, 4])
def test_p2p_between_gpus(al, staged, p):
    test_device_paths.test_p2p_ring_of_slots_and_rendezvous_into_registered_buffers(al, p)
    test_device_paths.test_p2p_small_messages_travel_as_packets(al, min(p, 3))
    comm = al.DeviceComm(emulate=p)
    test_device_emulated.test_p2p_sendrecv_ring(comm)
    test_device_emulated.test_p2p_in_place_exchange(comm)
    assert comm.stats()["local"] == 0
    comm.close()


@pytest.mark.parametrize("shape", [(1, 1, 1, 1, 1), (2, 3, 2, 5, 7), (1, 32, 4, 17, 19), (1, 5, 3, 64, 48), (1, 2, 16, 256, 252), (3, 1, 2, 300, 299)])
def test_halo_equals_flags(al, shape):
    from aluminum_b200.ops import HaloExchange
    n, c, d, h, w = shape
    for p, depth, periodic in ((2, 1, False), (2, 1, True), (4, 1, False), (3, min(2, d), True), (8, d, True), (4, d + 1, False)):
        comm = al.DeviceComm(emulate=p)
        comm.set_timeout_ms(3000)
        hx = HaloExchange(comm, n, c, d, h, w, depth, periodic)

        def call():
            for r, t in enumerate(hx.tensors):
                t.copy_(values(t.numel(), torch.float32, r).view(t.shape))
            hx.exchange()
            return [t.clone() for t in hx.tensors]
        if depth <= d:
            same(*both(al, comm, call))
        else:     # halos wider than the interior: the neighbour's planes are not all its own
            before = comm.stats()["local"]
            call()
            assert comm.stats()["local"] == before
        comm.close()


def test_halo_between_gpus(al, staged):
    from test_device_misc import test_halo_exchange_emulated
    test_halo_exchange_emulated(al)


@pytest.mark.parametrize("p", [2, 3, 8])
@pytest.mark.parametrize("dtype,op", [(torch.float32, "sum"), (torch.bfloat16, "avg"), (torch.float16, "max"), (torch.int32, "sum"), (torch.float64, "min")])
def test_small_operations(al, p, dtype, op):
    """At every size between buffers unless the packets' limits were set."""
    comm = al.DeviceComm(emulate=p)
    for n in (1, 2, 5, 64, 1023, 70001):
        for shift in (0, 1):
            def call():
                xs = [values(n, dtype, r, shift) for r in range(p)]
                outs = [torch.zeros(n + 2, dtype=dtype, device="cuda") for _ in range(p)]
                comm.allreduce(xs, [o[:n] for o in outs], op)
                comm.allreduce(xs, op=op)
                full = [values(p * n, dtype, r, shift) for r in range(p)]
                part = [torch.zeros(n + 2, dtype=dtype, device="cuda") for _ in range(p)]
                comm.reduce_scatter(full, [o[:n] for o in part], op)
                moved = [torch.zeros(p * n + 2, dtype=dtype, device="cuda") for _ in range(p)]
                comm.alltoall(full, [o[:p * n] for o in moved])
                every = [torch.zeros(p * n + 2, dtype=dtype, device="cuda") for _ in range(p)]
                comm.allgather(xs, [o[:p * n] for o in every])
                return outs + xs + part + moved + every
            same(*both(al, comm, call, 5))
    comm.close()


@pytest.mark.parametrize("name", ["ll_max_bytes", "ar_ll_max_bytes", "ar_ll2_max_bytes"])
def test_packet_limits_that_are_set(al, name):
    """Obeyed while one differs from its default; a value written back changes nothing, and defaults in their places end it."""
    comm, keep = al.DeviceComm(emulate=4), {row: al.get_tuning(f"{name}@{row}") for row in (2, 4, 8)}
    xs = [torch.ones(5, device="cuda") for _ in range(4)]

    def route():
        before = comm.stats()
        comm.allreduce(xs)
        return [k for k in ("ll", "local") if comm.stats()[k] > before[k]]
    assert route() == ["local"] and "packet_limits_set = 0" in al.info()
    for row, v in keep.items():
        al.set_tuning(f"{name}@{row}", v)
    assert route() == ["local"]
    for row in (2, 4, 8):
        try:
            al.set_tuning(f"{name}@{row}", keep[row] + 4096)
            assert route() == ["ll"] and "packet_limits_set = 1" in al.info()
        finally:
            al.set_tuning(f"{name}@{row}", keep[row])
        assert route() == ["local"]
    comm.close()


@pytest.mark.parametrize("n", [3, 700_001])
def test_movement_with_a_wire_type_is_not_taken(al, n):
    """Its counts are elements, not bytes: it stays with the staged kernels."""
    p = 4
    comm = al.DeviceComm(emulate=p)

    def call():
        xs, full = ([values(m, torch.float32, r) for r in range(p)] for m in (n, p * n))
        every, moved = ([torch.zeros(p * n, device="cuda") for _ in range(p)] for _ in range(2))
        comm.allgather(xs, every, wire_dtype=torch.bfloat16)
        comm.alltoall(full, moved, wire_dtype=torch.bfloat16)
        return every + moved
    same(*both(al, comm, call, 0))
    comm.close()
