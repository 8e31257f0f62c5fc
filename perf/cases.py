"""What this library's users have it do on one GPU, as cases that can be timed.

Two kinds of work.  The collective, row-exchange, point-to-point and halo kernels run with every rank of a
communicator on this GPU (``DeviceComm(emulate=p)``: the kernels and the flag protocol of the one-rank-per-GPU form,
one launch for all ranks).  The data-parallel trainer runs as one rank: forward, backward and the fused optimizer.

Every case is a plain dict; ``kind`` selects the family:

allreduce   one allreduce of ``n`` elements per rank; ``inplace`` runs it the way the gradient buckets do (in place,
            scaled by 1/p, non-blocking and joined), ``wire`` "bfloat16" halves what crosses the links
seqpar      a sequence-parallel layer's pair: reduce_scatter of a full activation, then allgather of a shard
ulysses     sequence -> head row exchange before attention and head -> sequence after it
experts     token dispatch to the rank of the chosen expert and the combine back, with uneven routing
halo        halo exchange of a 3-D tensor split along its depth
ring        every rank passes a block to the next one (ring attention, pipelines)
resnet      one ResNet-50 training step: bf16 autocast, cross entropy, fused momentum SGD
"""
import math

import torch

import aluminum_b200 as al
from aluminum_b200.models import resnet50
from aluminum_b200.ops import HaloExchange
from aluminum_b200.parallel import DataParallel, Trainer
from aluminum_b200.parallel import context, expert, ulysses

ESIZE = {"float32": 4, "bfloat16": 2, "float16": 2, "int32": 4}


def listed():
    return [
        # a loss, a gradient norm, a flag: nothing but latency
        {"name": "allreduce_1k", "kind": "allreduce", "p": 8, "n": 256, "dtype": "float32", "wire": "", "inplace": False},
        # a small layer's gradient on its own, length not a multiple of a vector
        {"name": "allreduce_600k_odd", "kind": "allreduce", "p": 4, "n": 300001, "dtype": "bfloat16", "wire": "", "inplace": False},
        # one 25 MB gradient bucket of the data-parallel trainer
        {"name": "bucket_25m", "kind": "allreduce", "p": 4, "n": 6553600, "dtype": "float32", "wire": "", "inplace": True},
        # the last, partly filled bucket with bf16 on the links
        {"name": "bucket_wire_bf16", "kind": "allreduce", "p": 8, "n": 3000009, "dtype": "float32", "wire": "bfloat16", "inplace": True},
        # sequence-parallel layer, 2048 x 4096 activations over 8 ranks
        {"name": "seqpar_2048x4096", "kind": "seqpar", "p": 8, "rows": 2048, "width": 4096, "dtype": "bfloat16"},
        # the same for a long context, 16384 x 8192 over 4 ranks
        {"name": "seqpar_16384x8192", "kind": "seqpar", "p": 4, "rows": 16384, "width": 8192, "dtype": "bfloat16"},
        # 8192 tokens of 32 heads x 128, sequence-sharded over 8 ranks
        {"name": "ulysses_8k", "kind": "ulysses", "p": 8, "s": 1024, "heads": 32, "d": 128, "dtype": "bfloat16"},
        # 4099 tokens per rank, width 2048, to the experts of 4 ranks
        {"name": "experts_4k", "kind": "experts", "p": 4, "tokens": 4099, "width": 2048, "dtype": "bfloat16"},
        # 3-D convolution slab: 32 channels, 16 planes of 256 x 256 per rank
        {"name": "halo_256", "kind": "halo", "p": 4, "c": 32, "d": 16, "h": 256, "w": 256, "depth": 1, "periodic": False},
        # key / value block of a context-parallel ring, 24 MiB and a ragged tail
        {"name": "ring_24m", "kind": "ring", "p": 4, "n": 12583001, "dtype": "bfloat16"},
        # the benchmark's training step
        {"name": "resnet50_b256", "kind": "resnet", "batch": 256},
        # fine tuning on small batches: many short kernels
        {"name": "resnet50_b24", "kind": "resnet", "batch": 24},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["allreduce", "allreduce", "allreduce", "seqpar", "seqpar", "ulysses", "experts", "halo", "ring", "resnet"])
    p = rng.choice([2, 3, 4, 8])
    if kind == "allreduce":
        inplace = rng.random() < 0.5
        wire = "bfloat16" if inplace and rng.random() < 0.3 else ""
        dtype = "float32" if inplace else rng.choice(["float32", "bfloat16", "float16", "int32"])
        return {"kind": kind, "p": p, "n": _log(rng, 2, 16 << 20), "dtype": dtype, "wire": wire, "inplace": inplace}
    if kind == "seqpar":
        p = rng.choice([2, 4, 8])
        return {"kind": kind, "p": p, "rows": p * _log(rng, 1, 2048), "width": _log(rng, 512, 8192),
                "dtype": rng.choice(["bfloat16", "float32"])}
    if kind == "ulysses":
        p = rng.choice([2, 4, 8])
        return {"kind": kind, "p": p, "s": _log(rng, 16, 2048), "heads": p * rng.randint(1, 6), "d": rng.choice([64, 80, 96, 128]),
                "dtype": "bfloat16"}
    if kind == "experts":
        return {"kind": kind, "p": p, "tokens": _log(rng, 64, 8192), "width": rng.choice([512, 1024, 1536, 2048, 4096]),
                "dtype": rng.choice(["bfloat16", "float32"])}
    if kind == "halo":
        return {"kind": kind, "p": p, "c": rng.randint(1, 32), "d": rng.randint(2, 16), "h": _log(rng, 17, 300),
                "w": _log(rng, 17, 300), "depth": rng.choice([1, 1, 2]), "periodic": rng.random() < 0.5}
    if kind == "ring":
        return {"kind": kind, "p": p, "n": _log(rng, 8, 24 << 20), "dtype": rng.choice(["bfloat16", "float32"])}
    return {"kind": kind, "batch": _log(rng, 8, 256)}


# ---------------------------------------------------------------------------------------------------------------------
def _values(gen, n, dtype):
    if not dtype.is_floating_point:
        return torch.randint(-1000, 1001, (n,), generator=gen, device="cuda", dtype=dtype)
    return torch.rand(n, generator=gen, device="cuda").mul_(2).sub_(1).to(dtype)


def prepare(case, seed):
    al.init()
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    st = dict(case)
    if kind == "resnet":
        torch.backends.cudnn.benchmark = True   # as bench.py sets it
        torch.manual_seed(seed)
        with torch.device("cuda"):
            model = resnet50().to(memory_format=torch.channels_last)
        dp = DataParallel(model, None, lr=0.1, momentum=0.9)
        # the running statistics as views of one buffer, so that a step's updated state comes back as one tensor
        bufs = [(m, k, getattr(m, k)) for m in model.modules() for k in ("running_mean", "running_var")
                if getattr(m, k, None) is not None]
        flat = torch.empty(sum(b.numel() for _, _, b in bufs), device="cuda")
        at = 0
        for m, k, b in bufs:
            view = flat[at:at + b.numel()]
            view.copy_(b)
            setattr(m, k, view)
            at += b.numel()
        st["trainer"], st["stats"] = Trainer(dp), flat
        st["x"] = torch.randn(case["batch"], 3, 224, 224, generator=gen, device="cuda")
        st["y"] = torch.randint(0, 1000, (case["batch"],), generator=gen, device="cuda")
        return st

    p = case["p"]
    comm = al.DeviceComm(emulate=p)
    st["comm"] = comm
    if kind == "halo":
        h = HaloExchange(comm, 1, case["c"], case["d"], case["h"], case["w"], case["depth"], case["periodic"])
        for t in h.tensors:
            t.uniform_(generator=gen)
        st["halo"] = h
        return st
    dtype = getattr(torch, case["dtype"])
    if kind == "allreduce":
        st["send"] = [_values(gen, case["n"], dtype) for _ in range(p)]
        st["recv"] = None if case["inplace"] else [torch.empty_like(x) for x in st["send"]]
        st["wire_dtype"] = getattr(torch, case["wire"]) if case["wire"] else None
    elif kind == "seqpar":
        n = case["rows"] * case["width"]
        st["full"] = [_values(gen, n, dtype) for _ in range(p)]
        st["shard"] = [_values(gen, n // p, dtype) for _ in range(p)]
        st["reduced"] = [torch.empty_like(x) for x in st["shard"]]
        st["gathered"] = [torch.empty_like(x) for x in st["full"]]
    elif kind == "ulysses":
        s, hd, d = case["s"], case["heads"], case["d"]
        st["x"] = [_values(gen, s * hd * d, dtype).view(s, hd, d) for _ in range(p)]
    elif kind == "experts":
        t, w = case["tokens"], case["width"]
        st["x"] = [_values(gen, t * w, dtype).view(t, w) for _ in range(p)]
        # uneven routing, rank 0's experts being the popular ones; which token goes where depends on the seed
        load = torch.linspace(0, 1, t, device="cuda").pow_(1.5).mul_(p).long().clamp_(max=p - 1)
        st["dest"] = [load[torch.randperm(t, generator=gen, device="cuda")] for _ in range(p)]
    elif kind == "ring":
        st["send"] = [_values(gen, case["n"], dtype) for _ in range(p)]
        st["recv"] = [torch.empty_like(x) for x in st["send"]]
    return st


def run(st):
    kind = st["kind"]
    if kind == "resnet":
        loss = st["trainer"].step_device(st["x"], st["y"])
        dp = st["trainer"].dp
        # the momentum is not returned on its own: with a zero-initialised branch scale the branches' gradients are
        # differences that bf16 rounding shifts by 2-4 % when nothing but the order of the images changes; the updated
        # parameters carry it at its weight in the step
        return {"loss": loss, "param": dp.flat_param, "stats": st["stats"]}
    comm = st["comm"]
    if kind == "allreduce":
        if st["inplace"]:
            req = comm.allreduce(st["send"], scale=1.0 / comm.size, wire_dtype=st["wire_dtype"], nonblocking=True)
            req.wait()
            return st["send"]
        comm.allreduce(st["send"], st["recv"])
        return st["recv"]
    if kind == "seqpar":
        comm.reduce_scatter(st["full"], st["reduced"])
        comm.allgather(st["shard"], st["gathered"])
        return {"reduced": st["reduced"], "gathered": st["gathered"]}
    if kind == "ulysses":
        heads = ulysses.seq_to_head(comm, st["x"])
        return {"heads": heads, "back": ulysses.head_to_seq(comm, heads)}
    if kind == "experts":
        got, state = expert.dispatch(comm, st["x"], st["dest"])
        return {"tokens": got, "back": expert.combine(comm, got, state)}
    if kind == "halo":
        st["halo"].exchange()
        return st["halo"].tensors
    context.ring_pass(comm, st["send"], st["recv"])
    return st["recv"]


def work(case):
    kind = case["kind"]
    if kind == "resnet":
        b = case["batch"]
        params = 25_557_032
        # 4.1 G multiply-adds per image forward, twice that backward; images and labels, parameters and momentum read and written
        return {"bytes": b * (3 * 224 * 224 * 4 + 8) + 4 * params * 4, "flops": b * 3 * 2 * 4.1e9}
    p = case["p"]
    if kind == "halo":
        pairs = p if case["periodic"] else p - 1
        slab = case["c"] * case["depth"] * case["h"] * case["w"] * 4
        return {"bytes": 2 * 2 * pairs * slab, "flops": 0}
    e = ESIZE[case["dtype"]]
    if kind == "allreduce":
        return {"bytes": 2 * p * case["n"] * e, "flops": (p - 1) * case["n"]}
    if kind == "seqpar":
        n = case["rows"] * case["width"]
        return {"bytes": (p * n + n + n + p * n) * e, "flops": (p - 1) * n}
    if kind == "ulysses":
        return {"bytes": 2 * 2 * p * case["s"] * case["heads"] * case["d"] * e, "flops": 0}
    if kind == "experts":
        return {"bytes": p * case["tokens"] * (2 * 2 * case["width"] * e + 8), "flops": 0}
    return {"bytes": 2 * p * case["n"] * e, "flops": 0}


def tolerance(case):
    kind = case["kind"]
    if kind == "resnet":
        # four times what permuting the images within the batch (another order of every sum) changes after two steps:
        # parameters 2.1e-4 / 0.05 at batch 8, 1.0e-4 / 0.02 at 24, 2.8e-5 / 0.006 at 256
        return {"rel": 2.4e-3 / math.sqrt(case["batch"]), "max": 0.57 / math.sqrt(case["batch"])}
    if kind in ("allreduce", "seqpar"):
        if case["dtype"] == "int32":
            return "exact"
        if case["dtype"] == "float32" and not case.get("wire"):
            return {"rel": 4e-7, "max": 2e-6}      # order of at most 8 fp32 additions (5e-8 from 64-bit sums)
        return {"rel": 8e-3, "max": 3e-2}          # one or two roundings to 16 bits (2.2e-3 from 64-bit sums)
    return "exact"


def exact(case, seed):
    """What ``run`` returns for these inputs from sums in 64 bits; None where outputs are copies (compared bit by bit)
    or follow a whole mixed-precision network."""
    kind = case["kind"]
    if kind not in ("allreduce", "seqpar") or case["dtype"] == "int32":
        return None
    p, dtype = case["p"], getattr(torch, case["dtype"])
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n = case["n"] if kind == "allreduce" else case["rows"] * case["width"]
    total = torch.zeros(n, dtype=torch.float64, device="cuda")
    for _ in range(p):                              # the draws of prepare(), in its order
        total += _values(gen, n, dtype).double()
    if kind == "allreduce":
        if case["inplace"]:
            total /= p
        return [total for _ in range(p)]
    return {"reduced": list(total.view(p, n // p)), "gathered": None}
