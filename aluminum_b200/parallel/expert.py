"""Expert parallelism: token dispatch to the rank that owns the chosen expert and the inverse combine.

Both directions are one row exchange (kernels/rows.cu): dispatch reads the tokens through the sort
permutation inside the kernel's publish step (no gather into a packed send buffer) and combine writes the
returning tokens through the same permutation in its consume step (no scatter afterwards).  The per-peer
token counts are exchanged with a small alltoall and read back with ONE device-to-host copy (the sizes of
the receive buffer have to be known on the host to allocate it); with all ranks in this process the routing kernel
leaves them in pinned memory that the host polls.
"""
from __future__ import annotations

import ctypes as C

import torch

from .. import _lib
from .._lib import AlError, check
from ._util import call, empties, unwrap, wrap


def _prefix(counts):
    out, run = [], 0
    for c in counts:
        out.append(run)
        run += c
    return out


_INTS = (torch.int64, torch.int32, torch.int16, torch.int8, torch.uint8)


def _on_device(comm, what, tensors):
    """Kernels get plain addresses: one tensor per local rank, all on the communicator's GPU."""
    if len(tensors) != comm.nlocal:
        raise AlError(f"{what}: expected {comm.nlocal} tensor(s), one per local rank, got {len(tensors)}")
    for t in tensors:
        if t.get_device() != comm.device_index:   # (-1 for host memory)
            raise AlError(f"{what}: must be on the communicator's GPU (cuda:{comm.device_index}), not on {t.device}")


# The routing kernel has one block per rank, all ranks at once: 25 us and (0.47 + 0.09 p) us per 1000 tokens.  A sort and a count take
# 95 to 200 us a rank, one rank after the other, and little more for more tokens.  One rank, kernel / sort in us: p = 2, 131072 tokens
# 106 / 155, 262144 tokens 186 / 158; p = 4, 131072 121 / 147, 262144 221 / 159; p = 8, 65536 102 / 143, 131072 176 / 143.
# Sorted from tokens * (p + 2) > this, per local rank, on.
_SORT_FROM = 950_000


def _sorted_route(d, p, counts):
    """The same order and counts by a sort (-1 counts where a destination is none of the p ranks)."""
    values, order = torch.sort(d, stable=True)
    first = torch.searchsorted(values, torch.arange(p + 1, device=d.device))
    good = (first[0] == 0) & (first[p] == d.numel())
    counts.copy_(torch.where(good, first[1:] - first[:-1], -1))
    return order


def _route(comm, dests, read=False):
    """Stable order of every local rank's tokens by destination, and a (2, local ranks, ranks) buffer whose first half
    holds the tokens per destination (one launch for all local ranks).  With ``read`` that half as lists instead, as soon as the
    launch has them."""
    n, p = len(dests), comm.size
    dests = list(dests)
    _on_device(comm, "dest_rank", dests)
    for r, d in enumerate(dests):
        if d.dim() != 1 or d.dtype not in _INTS:
            raise ValueError("dest_rank: a one-dimensional integer tensor per rank")
        if d.dtype != torch.int64 or not d.is_contiguous():
            dests[r] = d.to(torch.int64).contiguous()
    sizes = [d.numel() for d in dests]
    both = torch.empty((2, n, p), device=dests[0].device, dtype=torch.int64)
    if max(sizes) * (p + 2) > _SORT_FROM * n:
        order = [_sorted_route(d, p, c) for d, c in zip(dests, both[0].unbind())]
        return order, both[0].tolist() if read else both
    order = empties(comm, dests, [(s,) for s in sizes])
    args = (comm._h, n, (C.c_void_p * n)(*[d.data_ptr() for d in dests]), (C.c_size_t * n)(*sizes),
            (C.c_void_p * n)(*[o.data_ptr() for o in order]), both.data_ptr())
    if read:
        counts = (C.c_longlong * (n * p))()
        check(_lib.load().al_route_rows_read(*args, counts, comm._stream()))
        return order, [counts[r * p:(r + 1) * p] for r in range(n)]
    check(_lib.load().al_route_rows(*args, comm._stream()))
    return order, both


def dispatch(comm, tokens, dest_rank):
    """Send every token (row of ``tokens``) to ``dest_rank[i]``.

    Returns (received tokens grouped by source rank, state for :func:`combine`)."""
    p = comm.size
    toks = [t.contiguous() for t in wrap(comm, tokens)]
    dests = wrap(comm, dest_rank)
    _on_device(comm, "tokens", toks)
    for t, d in zip(toks, dests):
        if d.numel() > t.shape[0]:
            raise ValueError("dispatch: dest_rank has more entries than there are tokens")
    if comm.nlocal == p:     # every rank's counts are here
        order, sc = _route(comm, dests, read=True)
        rc = [list(col) for col in zip(*sc)]
    else:
        order, both = _route(comm, dests)
        call(comm, comm.alltoall, list(both[0].unbind()), list(both[1].unbind()))
        sc, rc = both.tolist()   # the one host read
    if any(c < 0 for row in sc + rc for c in row):
        raise ValueError(f"dest_rank: every destination must be a rank from 0 to {p - 1}")
    width = toks[0].shape[1]
    rb = width * toks[0].element_size()
    outs = empties(comm, [toks[0]] * len(rc), [(sum(r), width) for r in rc])
    one = comm.nlocal == 1
    zeros = [[0] * p for _ in sc]
    sf = [_prefix(r) for r in sc]
    rf = [_prefix(r) for r in rc]
    pick = (lambda t: t[0]) if one else (lambda t: t)
    comm.exchange_rows(pick(toks), pick(outs), rb, rb, rb, pick(sc), pick(sf), pick(zeros), pick(rc), pick(rf),
                       pick(zeros), send_idx=pick(order))
    state = {"order": order, "sc": sc, "sf": sf, "rc": rc, "rf": rf, "width": width, "like": tokens}
    return unwrap(comm, outs, tokens), state


def combine(comm, expert_out, state):
    """Return processed tokens to the ranks (and positions) they came from."""
    p = comm.size
    outs_in = [t.contiguous() for t in wrap(comm, expert_out)]
    width = state["width"]
    rb = width * outs_in[0].element_size()
    one = comm.nlocal == 1
    # directions swap: what was received is sent back, and lands through the sort permutation
    sc, sf, rc, rf = state["rc"], state["rf"], state["sc"], state["sf"]
    back = empties(comm, [outs_in[0]] * len(rc), [(sum(r), width) for r in rc])
    zeros = [[0] * p for _ in sc]
    pick = (lambda t: t[0]) if one else (lambda t: t)
    comm.exchange_rows(pick(outs_in), pick(back), rb, rb, rb, pick(sc), pick(sf), pick(zeros), pick(rc), pick(rf),
                       pick(zeros), recv_idx=pick(state["order"]))
    return unwrap(comm, back, state["like"])
