"""The work whose speed matters to a user of this framework, as cases that can be timed on
one GPU.  A case is a dict of plain values; `prepare` makes what a program has in hand
before the call, `run` makes one pass through the public entry points.

Five kinds of case:

* ``step``   the synchronisation of a whole model's gradients, once per training step
             (``DistributedOptimizer.synchronize``): every algorithm, both topologies
* ``bucket`` one flat gradient bucket handed over by a DDP communication hook or by a
             program's own hook (``FlatSyncer.sync_``)
* ``codec``  the decoupled primitives (``Compressor``) a program composes its own schedule
             from: ``roundtrip`` (encode at the sender, decode at the receiver), ``hop``
             (one ring hop: decode the incoming payload, merge, encode) and ``serve`` (a
             parameter server: decode-accumulate the payloads of the ranks, encode the sum)
* ``generated``  an encode / decode pair generated from its DSL source

With one GPU a job has one rank: the fused kernels still encode, hand over through the
inbox, and decode.  Gradients are synchronised in place, so from the second pass on the
gradient is the previous result, as with a constant gradient in training.
"""
import math
import random

import torch

import hipress_b200 as hp
from hipress_b200.compll import load_op
from hipress_b200.config import HipressConfig
from hipress_b200.models import get_model
from hipress_b200.parallel.hooks import FlatSyncer

ALGORITHMS = ("onebit", "tbq", "terngrad", "dgc", "graddrop")
SPARSE = ("dgc", "graddrop")


def listed():
    return [
        # a small model: a few microseconds of GPU work, so launches and the host path
        # decide (MLP 784-256-10, the smallest training configuration)
        {"name": "step mlp tbq ring", "kind": "step", "model": "mlp", "algorithm": "tbq", "topology": "ring",
         "comp_threshold": 1024},
        # the headline configurations: VGG-19 + TBQ + ring, ResNet-50 + DGC + PS, BERT + onebit
        # + ring (the base model: large shards of the same shapes), and a sequence model
        # with stochastic rounding through PS
        {"name": "step vgg19 tbq ring", "kind": "step", "model": "vgg19", "algorithm": "tbq", "topology": "ring",
         "comp_threshold": 262144},
        {"name": "step resnet50 dgc ps", "kind": "step", "model": "resnet50", "algorithm": "dgc", "topology": "ps",
         "comp_threshold": 262144},
        {"name": "step bert_base onebit ring", "kind": "step", "model": "bert_base", "algorithm": "onebit",
         "topology": "ring", "comp_threshold": 262144},
        {"name": "step transformer terngrad ps", "kind": "step", "model": "transformer", "algorithm": "terngrad",
         "topology": "ps", "comp_threshold": 262144},
        # DDP's default bucket (25 MB of fp32) through the communication hook's path
        {"name": "bucket 25MB graddrop ring", "kind": "bucket", "n": 6553600, "algorithm": "graddrop",
         "topology": "ring", "ratio": 0.001},
        # one small layer: the latency of the smallest calls
        {"name": "codec terngrad 2bit small", "kind": "codec", "op": "roundtrip", "n": 2560,
         "algorithm": "terngrad", "bits": 2},
        # an embedding-sized layer with 8-bit codes: the widest payload, memory bound
        {"name": "codec terngrad 8bit 256MB", "kind": "codec", "op": "roundtrip", "n": 67108864,
         "algorithm": "terngrad", "bits": 8},
        # one hop of a ring made of primitives, ragged length
        {"name": "codec tbq hop 64MB", "kind": "codec", "op": "hop", "n": 16777213, "algorithm": "tbq", "bits": 2},
        # a parameter server that sums four ranks' payloads of a medium layer, ragged length
        {"name": "codec onebit serve 4MB", "kind": "codec", "op": "serve", "n": 1048583, "algorithm": "onebit",
         "bits": 1},
        # exact top-0.1 % with momentum correction of a medium layer
        {"name": "codec dgc 4MB", "kind": "codec", "op": "roundtrip", "n": 1000003, "algorithm": "dgc",
         "ratio": 0.001},
        # the generator's output for a function with a whole-tensor reduction
        {"name": "generated terngrad 64MB", "kind": "generated", "n": 16777216, "algorithm": "terngrad", "bits": 2},
    ]


def _log_size(rng, lo, hi):
    return max(1, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choices(("step", "bucket", "codec", "generated"), (6, 3, 8, 2))[0]
    alg = rng.choice(ALGORITHMS)
    c = {"kind": kind, "algorithm": alg}
    if kind == "step":
        # a generic model: some tensors of very different sizes, small ones below the threshold
        tensors, elements = rng.randint(1, 24), _log_size(rng, 3e4, 2.5e7 if alg in SPARSE else 8e7)
        c.update(topology=rng.choice(("ring", "ps")), tensors=tensors, elements=elements, split=rng.randrange(1 << 20),
                 # at most the mean size, so that at least one tensor is compressed
                 comp_threshold=rng.choice([t for t in (1024, 16384, 262144) if t <= max(1024, elements // tensors)]))
    elif kind == "bucket":
        c.update(topology=rng.choice(("ring", "ps")), n=_log_size(rng, 1e4, 2e7 if alg in SPARSE else 6e7))
    elif kind == "codec":
        op = "roundtrip" if alg in SPARSE else rng.choice(("roundtrip", "roundtrip", "hop", "serve"))
        c.update(op=op, n=_log_size(rng, 1e3, 2e7 if alg in SPARSE else (3e7 if op == "serve" else 6e7)))
    else:
        c["algorithm"] = alg = rng.choice(("onebit", "tbq", "terngrad"))
        c.update(n=_log_size(rng, 1e4, 3e7))
    if alg in SPARSE:
        c["ratio"] = rng.choice((0.001, 0.001, 0.01))
    elif kind != "step":
        c["bits"] = {"onebit": 1, "tbq": 2}.get(alg) or rng.choice((1, 2, 4, 8))
    return c


# ------------------------------------------------------------------- inputs
def _gradient(n, gen):
    """Gradient values: centred, heavy-tailed, of the size TBQ's default threshold is made for."""
    g = torch.randn(n, device="cuda", generator=gen)
    return g.mul_(torch.randn(n, device="cuda", generator=gen)).mul_(0.01)


def _shapes(case):
    """(name, element count) of the model's parameters."""
    if case.get("model") == "mlp":
        return [("fc1.weight", 256 * 784), ("fc1.bias", 256), ("fc2.weight", 10 * 256), ("fc2.bias", 10)]
    if "model" in case:
        with torch.device("meta"):
            m = get_model(case["model"])
        return [(n, p.numel()) for n, p in m.named_parameters()]
    rng = random.Random(case["split"])
    w = [math.exp(rng.uniform(0.0, 7.0)) for _ in range(case["tensors"])]
    return [("p%d" % i, max(1, int(case["elements"] * x / sum(w)))) for i, x in enumerate(w)]


def _algorithm_options(case):
    kw = {}
    if "ratio" in case:
        kw["ratio"] = case["ratio"]
    if case["algorithm"] == "terngrad" and "bits" in case:
        kw["bitwidth"] = case["bits"]
    return kw


def prepare(case, seed):
    hp.init()
    gen = torch.Generator("cuda").manual_seed(seed)
    kind, alg = case["kind"], case["algorithm"]
    st = {"kind": kind}
    if kind == "step":
        # parameters whose gradients lie in one buffer, each on a 256-byte boundary
        shapes = _shapes(case)
        starts, total = [], 0
        for _, n in shapes:
            starts.append(total)
            total += (n + 63) // 64 * 64
        flat = _gradient(total, gen)
        named = []
        for (name, n), lo in zip(shapes, starts):
            p = torch.nn.Parameter(torch.zeros(n, device="cuda"))
            p.grad = flat[lo:lo + n]
            named.append((name, p))
        opt = hp.DistributedOptimizer(torch.optim.SGD([p for _, p in named], lr=0.01), named, algorithm=alg,
                                      topology=case["topology"], comp_threshold=case["comp_threshold"],
                                      **_algorithm_options(case))
        st.update(opt=opt, grads=flat, named=named,
                  state=[list(e.state.values()) for e in opt.engine.entries if e.state])
    elif kind == "bucket":
        cfg = HipressConfig(algorithm=alg, topology=case["topology"], comp_threshold=0, **_algorithm_options(case))
        st.update(syncer=FlatSyncer(cfg), flat=_gradient(case["n"], gen))
    elif kind == "codec":
        n = case["n"]
        c = hp.Compressor(alg, **_algorithm_options(case))
        g = [_gradient(n, gen)]
        if c.spec.sparse:
            # successive gradients that cancel, as noise does: under one constant gradient an
            # accumulator only ever grows, and the selection would see a state training never has
            h = _gradient(n, gen)
            g += [-g[0], h, -h]
        st.update(op=case["op"], comp=c, g=g, turn=0, state=c.new_state(n, "cuda"),
                  ws=c.new_workspace("cuda", n), payload=torch.zeros(c.payload_bytes(n), dtype=torch.uint8, device="cuda"),
                  out=torch.zeros(n, device="cuda"))
        for r in st["state"].values():     # what earlier steps left behind
            r.copy_(_gradient(n, gen))
        if case["op"] in ("hop", "serve"):
            peers = 1 if case["op"] == "hop" else 4
            st["incoming"] = []
            for q in range(peers):
                st["incoming"].append(c.encode(_gradient(n, gen), c.new_state(n, "cuda"), step=3, salt=q))
    else:
        n, bits = case["n"], case["bits"]
        stem = {"onebit": "Onebit", "tbq": "Tbq", "terngrad": "TernGrad"}[alg]
        head = 10 if alg == "terngrad" else 4
        st.update(algorithm=alg, bits=bits, g=_gradient(n, gen), residual=_gradient(n, gen),
                  payload=torch.zeros(head + (n * bits + 7) // 8, dtype=torch.uint8, device="cuda"),
                  out=torch.zeros(n, device="cuda"), encode=load_op(stem + "Encode"), decode=load_op(stem + "Decode"))
    return st


# --------------------------------------------------------------------- passes
def run(st):
    kind = st["kind"]
    if kind == "step":
        st["opt"].synchronize()
        return {"grads": st["grads"], "state": st["state"]}
    if kind == "bucket":
        st["syncer"].sync_(st["flat"])
        return {"flat": st["flat"], "state": list(st["syncer"].state[0][0].values())}
    if kind == "codec":
        c, op = st["comp"], st["op"]
        g = st["g"][st["turn"] % len(st["g"])]
        st["turn"] += 1
        if op == "roundtrip":
            c.encode(g, st["state"], out=st["payload"], step=7, tensor_id=1, workspace=st["ws"])
            c.decode(st["payload"], st["out"])
            # pairs of a top-k payload come in no particular order: what it says is in `out`
            return {"payload": None if c.spec.sparse else st["payload"], "out": st["out"], "state": st["state"]}
        if op == "hop":
            c.encode(g, st["state"], incoming=st["incoming"][0], out=st["payload"], step=7, tensor_id=1)
            return {"payload": st["payload"], "state": st["state"]}
        for q, p in enumerate(st["incoming"]):
            c.decode(p, st["out"], accumulate=q > 0)
        c.encode(st["out"], st["state"], out=st["payload"], step=7, tensor_id=1)
        return {"payload": st["payload"], "sum": st["out"], "state": st["state"]}
    if st["algorithm"] == "tbq":
        st["encode"](st["g"], st["residual"], st["payload"], 0.01)
    elif st["algorithm"] == "onebit":
        st["encode"](st["g"], st["residual"], st["payload"])
    else:
        st["encode"](st["g"], st["payload"], st["bits"], seed=1)
    st["decode"](st["payload"], st["out"])
    return {"payload": st["payload"], "out": st["out"], "residual": st["residual"]}


# ----------------------------------------------------------------------- work
def work(case):
    alg, kind = case["algorithm"], case["kind"]
    # bytes of per-rank state an encode reads and writes, per element
    state = {"onebit": 8, "tbq": 8, "terngrad": 0, "dgc": 16, "graddrop": 8}[alg]
    if kind in ("step", "bucket"):
        n = sum(x for _, x in _shapes(case) if x >= case["comp_threshold"]) if kind == "step" else case["n"]
        b = 8 + state           # gradient in, average out, state
        if case["topology"] == "ps" and alg != "terngrad":
            b += 4 if alg in SPARSE else 8      # the owner's state: read, and written when dense
        return {"bytes": float(max(n, 1) * b), "flops": float(8 * max(n, 1))}
    n = case["n"]
    if alg in SPARSE:
        pairs = 8.0 * math.ceil(n * case["ratio"])
        return {"bytes": n * (4.0 + state) + 4.0 * n + 2 * pairs, "flops": 6.0 * n}
    code = n * case["bits"] / 8.0
    if kind == "generated":         # encode: gradient (and residual) in, codes out; decode: codes in, values out
        return {"bytes": n * (4.0 + state) + 4.0 * n + 2 * code, "flops": 8.0 * n}
    if case["op"] == "roundtrip":
        return {"bytes": n * (4.0 + state) + 4.0 * n + 2 * code, "flops": 8.0 * n}
    if case["op"] == "hop":
        return {"bytes": n * (4.0 + state) + 2 * code, "flops": 8.0 * n}
    return {"bytes": n * (4.0 + state) + 5 * code, "flops": 16.0 * n}     # the sum is written once, then encoded


def tolerance(case):
    if case["algorithm"] == "onebit":
        # the scale is a sum: its last bit may differ with the order of the additions, and
        # with it the bytes that hold it
        return {"rel": 1e-5, "differ": 1e-3 if case.get("n", 1 << 20) < 1 << 16 else 1e-5}
    if case["algorithm"] in SPARSE:
        return {"rel": 1e-6}    # plain fp32 multiply-adds and copies
    return "exact"              # thresholds, integer draws and codes: nothing to round differently
