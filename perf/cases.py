"""The work a program has this package do, as cases that can be timed.

Four families, all through the public classes, on one GPU:

* ``exchange``: one compressed message of a ``Comprex`` engine: ``writeRemote`` of a fresh vector with
  error feedback, ``readRemote_add`` or ``readRemote`` on the receiving side.  The engine is connected
  to its own rank, so both halves run.  Sizes, top-k fractions and element types are those of the
  allreduce sweep (2^16 to 2^28 elements, 0.1 / 1 / 10 %, fp32 and bf16 vectors); ``exact`` takes the
  threshold from a select over the whole vector, ``codec`` is ``pairs`` or ``rle``.
* ``dense``: one dense message of a ``GaspiEx`` engine, added into the receiver's vector.
* ``bigring``: the compressed allreduce of one gradient bucket the way the DDP hook calls it (send half,
  then a receive half that writes the mean), for all ranks of a ``LoopbackWorld`` of ``ranks`` ranks.
* ``optimizer``: one ``apply_gradients`` of ``ComprexOptimizer`` on the parameters of a model of this
  package: LeNet-5, ResNet-50 and GPT-2 medium with the settings of the training benchmark, on one rank
  either with the exchange (``exchange`` true) or without it (the default of a single-rank job).
"""
import math

import torch

import comprex_b200 as cx
from comprex_b200.models.gpt2 import GPT2
from comprex_b200.models.lenet import LeNet5
from comprex_b200.models.resnet import ResNet
from comprex_b200.ops import primitives as P
from comprex_b200.optim import ComprexOptimizer

_DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16}
_BYTES = {"fp32": 4, "bf16": 2, "fp16": 2}


def listed():
    return [
        # the smallest vector of the sweep: threshold, compress and decode are all launch latency
        dict(name="exchange-64k", kind="exchange", n=1 << 16, dtype="fp32", ratio=0.01, codec="pairs", exact=False,
             read="add"),
        # the two-rank exchange configuration: 2^20 elements, top-k 1 %; the receiver wants the dense vector
        dict(name="exchange-1Mi", kind="exchange", n=1 << 20, dtype="fp32", ratio=0.01, codec="pairs", exact=False,
             read="set"),
        # all of ResNet-50's gradients as one bf16 vector (25 557 032 elements, not a multiple of 1024)
        dict(name="exchange-resnet-bf16", kind="exchange", n=25557032, dtype="bf16", ratio=0.001, codec="pairs",
             exact=False, read="add"),
        # the largest vector of the sweep
        dict(name="exchange-256Mi", kind="exchange", n=1 << 28, dtype="fp32", ratio=0.01, codec="pairs", exact=False,
             read="add"),
        # threshold selected over the whole vector instead of a sample; an odd length
        dict(name="exchange-exact-10M", kind="exchange", n=10000019, dtype="fp32", ratio=0.01, codec="pairs",
             exact=True, read="set"),
        # the run-length codec at the densest top-k of the sweep; an odd length
        dict(name="exchange-rle-4M", kind="exchange", n=4194301, dtype="fp32", ratio=0.1, codec="rle", exact=False,
             read="add"),
        # a dense bf16 message
        dict(name="dense-16Mi-bf16", kind="dense", n=1 << 24, dtype="bf16"),
        # one 25 MB fp32 gradient bucket of an eight-rank job (all eight ranks' work)
        dict(name="bigring-8x25MB", kind="bigring", n=6553600, dtype="fp32", ratio=0.01, ranks=8),
        # LeNet-5 step: ten small tensors
        dict(name="lenet-step", kind="optimizer", model="lenet", depth=0, width=0, vocab=10, dtype="fp32", rule="sgd",
             momentum=0.0, ratio=0.01, exchange=True),
        # ResNet-50 step of a single-rank job: clip, momentum and update, nothing to exchange
        dict(name="resnet50-step-local", kind="optimizer", model="resnet", depth=3, width=64, vocab=1000, dtype="bf16",
             rule="sgd", momentum=0.9, ratio=0.01, exchange=False),
        # ResNet-50 step with the compressed exchange, 25 MB buckets
        dict(name="resnet50-step", kind="optimizer", model="resnet", depth=3, width=64, vocab=1000, dtype="bf16",
             rule="sgd", momentum=0.9, ratio=0.01, exchange=True),
        # GPT-2 medium step with the compressed exchange and AdamW, 25 MB buckets, top-k 0.1 %
        dict(name="gpt2-medium-step", kind="optimizer", model="gpt2", depth=24, width=1024, vocab=50257, dtype="bf16",
             rule="adamw", momentum=0.0, ratio=0.001, exchange=True),
    ]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["exchange", "exchange", "exchange", "rle", "dense", "bigring", "optimizer", "optimizer"])
    ratio = rng.choice([0.001, 0.01, 0.1])
    dtype = rng.choice(["fp32", "bf16", "fp16"])
    if kind == "exchange":
        exact = rng.random() < 0.25
        n = _log_size(rng, 1 << 16, 1 << (25 if exact else 27))
        return dict(kind="exchange", n=n, dtype=dtype, ratio=ratio, codec="pairs", exact=exact,
                    read=rng.choice(["add", "set"]))
    if kind == "rle":
        return dict(kind="exchange", n=_log_size(rng, 1 << 16, 1 << 24), dtype=dtype, ratio=ratio, codec="rle",
                    exact=False, read=rng.choice(["add", "set"]))
    if kind == "dense":
        return dict(kind="dense", n=_log_size(rng, 1 << 16, 1 << 27), dtype=dtype)
    if kind == "bigring":
        return dict(kind="bigring", n=_log_size(rng, 1 << 16, 1 << 23), dtype=dtype, ratio=rng.choice([0.001, 0.01]),
                    ranks=rng.randint(2, 8))
    if rng.random() < 0.5:
        return dict(kind="optimizer", model="resnet", depth=rng.randint(1, 4), width=rng.choice([16, 24, 32, 48, 64]),
                    vocab=rng.randint(10, 1000), dtype=rng.choice(["fp32", "bf16"]), rule="sgd", momentum=0.9,
                    ratio=rng.choice([0.001, 0.01]), exchange=rng.random() < 0.5)
    return dict(kind="optimizer", model="gpt2", depth=rng.randint(2, 16), width=rng.choice([128, 256, 512, 768, 1024]),
                vocab=rng.randint(257, 50257), dtype=rng.choice(["fp32", "bf16"]), rule=rng.choice(["adamw", "sgd"]),
                momentum=0.9, ratio=rng.choice([0.001, 0.01]), exchange=rng.random() < 0.75)


# ---- states ---------------------------------------------------------------------------------------
def _gen(seed, k=0):
    return torch.Generator(device="cuda").manual_seed((int(seed) * 1000003 + k) % (1 << 62))


def _gauss(n, dtype, gen):
    return torch.randn(n, device="cuda", generator=gen).to(dtype)


class _Ranks:
    """A LoopbackWorld that is closed when the state goes."""

    def __init__(self, ranks):
        self.world = cx.LoopbackWorld(ranks, device="cuda")

    def __del__(self):
        self.world.close()


def _prepare_exchange(case, seed):
    env = cx.GaspiEnvironment(1 << 20, device="cuda")
    n, gen = case["n"], _gen(seed)
    engine = cx.Comprex(env, n, 1.0)
    engine.setThreshold(cx.ThresholdTopK(case["ratio"], exact=case["exact"]))
    engine.setCompressor(cx.CompressorRLE() if case["codec"] == "rle" else cx.CompressorIndexPairs())
    engine.connectTx(0)
    engine.connectRx(0)
    # gradients are N(0, 1); the residual is what earlier steps held back
    vec = _gauss(n, _DTYPES[case["dtype"]], gen)
    engine.setRests(torch.randn(n, device="cuda", generator=gen).mul_(0.5))
    out = torch.zeros(n, device="cuda")
    return dict(kind="exchange", engine=engine, vec=vec, out=out, add=case["read"] == "add")


def _prepare_dense(case, seed):
    env = cx.GaspiEnvironment(1 << 20, device="cuda")
    dt, gen = _DTYPES[case["dtype"]], _gen(seed)
    engine = cx.GaspiEx(env, case["n"], dt)
    engine.connectTx(0)
    engine.connectRx(0)
    return dict(kind="dense", engine=engine, vec=_gauss(case["n"], dt, gen), out=_gauss(case["n"], dt, gen))


def _prepare_bigring(case, seed):
    n, ranks, dt = case["n"], case["ranks"], _DTYPES[case["dtype"]]
    holder = _Ranks(ranks)
    reducers, grads, outs = [], [], []
    for r, env in enumerate(holder.world.envs):
        red = cx.Comprex_BigRingAllreduce(env)
        # room for five times the expected survivors: the sampled threshold is an estimate
        red.setup_connections(n, 1, case["ratio"], max(10.0 * case["ratio"], 0.05), consistent=True)
        reducers.append(red)
        grads.append(_gauss(n, dt, _gen(seed, r)))
        outs.append(torch.zeros(n, dtype=dt, device="cuda"))
    return dict(kind="bigring", holder=holder, reducers=reducers, grads=grads, outs=outs, scale=1.0 / ranks)


def _model(case):
    if case["model"] == "lenet":
        return LeNet5(case["vocab"])
    if case["model"] == "resnet":
        # depth 3 is the layer plan of ResNet-50
        layers = (3, 4, 6, 3) if case["depth"] == 3 else (case["depth"],) * 4
        return ResNet(layers, case["vocab"], case["width"]).to(memory_format=torch.channels_last)
    w = case["width"]
    return GPT2(case["depth"], w, max(w // 64, 1), 4 * w, case["vocab"], 1024)


def _prepare_optimizer(case, seed):
    torch.manual_seed(int(seed))
    with torch.device("cuda"):
        model = _model(case).to(_DTYPES[case["dtype"]])
    env = cx.GaspiEnvironment(1 << 20, device="cuda")
    if case["rule"] == "adamw":
        kw = dict(lr=3e-4, rule="adamw", weight_decay=0.1, betas=(0.9, 0.95))
    else:
        kw = dict(lr=0.01, momentum=case["momentum"], rule="sgd", weight_decay=0.0)
    opt = ComprexOptimizer(model.parameters(), env, compression_ratio=case["ratio"], bucket_cap_mb=25.0,
                           single_rank_bypass=not case["exchange"], **kw)
    gen = _gen(seed)
    pairs = []
    for i, p in enumerate(model.parameters()):
        # per-tensor gradient scales spread over two decades; the largest tensors exceed the clip norm
        scale = 10.0 ** (-3.0 + 2.0 * ((i * 7) % 11) / 10.0)
        pairs.append((torch.empty_like(p).normal_(0.0, scale, generator=gen), p))
    return dict(kind="optimizer", model=model, opt=opt, pairs=pairs, rule=case["rule"])


def prepare(case, seed):
    return {"exchange": _prepare_exchange, "dense": _prepare_dense, "bigring": _prepare_bigring,
            "optimizer": _prepare_optimizer}[case["kind"]](case, seed)


# ---- one pass -------------------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "exchange":
        engine, out = state["engine"], state["out"]
        engine.writeRemote(state["vec"])
        if state["add"]:
            engine.readRemote_add(out)
        else:
            engine.readRemote(out)
        return {"received": out, "rests": engine.getRests_p()}
    if kind == "dense":
        state["engine"].writeRemote(state["vec"])
        state["engine"].readRemote_add(state["out"])
        return {"received": state["out"]}
    if kind == "bigring":
        sent = [red.send_fast(g) for red, g in zip(state["reducers"], state["grads"])]
        for red, out, (seq, par) in zip(state["reducers"], state["outs"], sent):
            red.recv_fast(seq, par, P.args_set(out, state["scale"]))
        return {"mean": state["outs"], "rests": [red.rests for red in state["reducers"]]}
    opt = state["opt"]
    opt.apply_gradients(state["pairs"])
    res = {"master": opt._master, "rests": [ar.rests for ar in opt.comprex_allreducers.values()]}
    if opt._shadow is not None:
        res["weights"] = opt._shadow
    if state["rule"] == "adamw":
        res["m"], res["v"] = opt._m, opt._v
    else:
        res["momentum"] = opt._update
    return res


# ---- what a pass cannot do without ------------------------------------------------------------------
def _parameters(case):
    with torch.device("meta"):
        return sum(p.numel() for p in _model(case).parameters())


def work(case):
    """Every input read once and every output written once, the message written and read once.  Messages:
    8 bytes a pair; run-length: 4 bytes a value and two 4-byte runs for it."""
    kind, es = case["kind"], _BYTES[case["dtype"]]
    if kind == "dense":
        n = case["n"]
        return {"bytes": 5 * es * n, "flops": n}            # vector, message out and in, sum read and written
    if kind == "exchange":
        n, k = case["n"], case["ratio"] * case["n"]
        message = 2 * (12 if case["codec"] == "rle" else 8) * k
        return {"bytes": (es + 8) * n + message + (8 * k if case["read"] == "add" else 4 * n), "flops": 2 * n}
    if kind == "bigring":
        n, k, p = case["n"], case["ratio"] * case["n"], case["ranks"]
        return {"bytes": p * ((es + 8) * n + 16 * p * k + es * n), "flops": p * (2 * n + p * k)}
    n = _parameters(case)
    k, low = case["ratio"] * n, es if es < 4 else 0
    if case["rule"] == "adamw":
        # gradient, w / m / v read and written, low-precision weights written
        total = (es + 24 + low) * n + ((8 * n + 16 * k) if case["exchange"] else 0)
    elif case["exchange"]:
        # gradient, momentum, residual; only the addressed weights change
        total = (es + 8 + 8) * n + (16 + 8 + low) * k
    else:
        total = (es + 8 + 8 + low) * n
    return {"bytes": total, "flops": (15 if case["rule"] == "adamw" else 6) * n}


def tolerance(case):
    # sums of few fp32 terms; vectors and weights held in 16 bits round once per pass
    if case["kind"] in ("dense", "bigring", "optimizer") and case["dtype"] != "fp32":
        return {"rel": 1e-2}
    return {"rel": 1e-5}
