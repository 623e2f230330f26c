"""GaspiEx / Comprex / FastComprex on two (or three) virtual ranks of one device.

Scenarios follow the reference's own checks: test/comprex.cpp (3 x writeRemote +
flushRests, receiver accumulates with readRemote_add, result == 3 * values),
examples/comprEx.cpp, examples/gaspiEx.py.
"""
import math
import threading
import time

import numpy as np
import pytest
import torch

import comprex_b200 as cx

from helpers import alt_ramp, ref_threshold_topk


@pytest.fixture
def world(device):
    w = cx.LoopbackWorld(3, device=device, timeout_ms=300)
    yield w
    w.close()


def make(world, cls, *args, **kw):
    return [cls(e, *args, **kw) for e in world.envs]


def test_gaspiex_roundtrip_and_add(world):
    n, dev = 5003, world.device
    ex = make(world, cx.GaspiEx, n)
    ex[0].connectTx(1, 0)
    ex[1].connectRx(0, 0)
    for step in range(4):   # more messages than slots: parity reuse
        v = torch.randn(n, device=dev)
        ex[0].writeRemote(v)
        if step % 2 == 0:
            assert torch.equal(ex[1].readRemote(), v)
        else:
            acc = torch.ones(n, device=dev)
            ex[1].readRemote_add(acc)
            assert torch.equal(acc, v + 1)
    with pytest.raises(cx.ComprexError, match="too large"):
        ex[0].writeRemote(torch.zeros(n + 1, device=dev))
    with pytest.raises(cx.ComprexError, match="without connecting"):
        ex[2].writeRemote(torch.zeros(n, device=dev))


def test_gaspiex_numpy_vectors_and_short_messages(world):
    ex = make(world, cx.GaspiEx, 100)
    ex[0].connectTx(2, 5)
    ex[2].connectRx(0, 5)
    v = np.arange(60, dtype=np.float32)
    ex[0].writeRemote(v)
    out = np.zeros(60, dtype=np.float32)
    ex[2].readRemote_vec(out, 60)
    assert np.array_equal(out, v)


def test_gaspiex_broadcast_shared_buffer_and_forward(world):
    n, dev = 2000, world.device
    ex = make(world, cx.GaspiEx, n)
    v = torch.randn(n, device=dev)
    # chief 0 -> {1, 2} in one launch
    ex[0].writeRemote_multi(v, [1, 2])
    for r in (1, 2):
        ex[r].connectRx(0, 0)
        assert torch.equal(ex[r].readRemote(), v)
    # shared-buffer fan-out of the reference: second engine re-sends the first one's vector
    a, b = make(world, cx.GaspiEx, n), make(world, cx.GaspiEx, n)
    a[0].connectTx(1, 1)
    b[0].connectTx_sameBufferAs(2, 2, a[0])
    a[1].connectRx(0, 1)
    b[2].connectRx(0, 2)
    a[0].writeRemote(v)
    b[0].writeRemote(size=n)
    assert torch.equal(a[1].readRemote(), v) and torch.equal(b[2].readRemote(), v)
    # ring hop: 0 -> 1 -> 2 with forward_buffer / forward_add
    ring = make(world, cx.GaspiEx, n)
    ring[0].connectTx(1, 0)
    ring[1].connectTo(0, 2, 0)
    ring[2].connectRx(1, 0)
    ring[0].writeRemote(v)
    mid = torch.ones(n, device=dev)
    ring[1].readRemote_wait()
    ring[1].forward_buffer()
    ring[1].forward_add(mid)
    assert torch.equal(mid, v + 1)
    assert torch.equal(ring[2].readRemote(), v)


@pytest.mark.parametrize("n,topk", [(50, 0.1), (500000, 0.01)])
def test_comprex_write_flush_accumulate(world, n, topk):
    """test/comprex.cpp:73-120 and examples/comprEx.cpp: nothing is lost after flushRests."""
    dev = world.device
    cm = make(world, cx.Comprex, n, 3.0, True)
    for c in cm:
        c.setThreshold(cx.ThresholdTopK(topk))
        c.setCompressor(cx.CompressorIndexPairs())
    cm[0].connectTx(1, 1)
    cm[1].connectRx(0, 1)
    vals = alt_ramp(n, dev)
    acc = torch.zeros(n, device=dev)
    runs = 3
    for _ in range(runs):
        cm[0].writeRemote(vals)
        cm[1].readRemote_add(acc)
    assert not torch.equal(acc, runs * vals)            # something was held back ...
    held = cm[0].getRests()
    assert torch.equal(acc + held, runs * vals)          # ... and it sits in the residual
    cm[0].flushRests()
    cm[1].readRemote_add(acc)
    assert torch.equal(acc, runs * vals)
    assert float(cm[0].getRests().abs().sum()) == 0.0
    st = cm[0].stats()
    assert st["n"] == n and st["status"] == 0


def test_comprex_topk_fraction_and_threshold_readback(world):
    n, dev = 1 << 18, world.device
    cm = make(world, cx.Comprex, n, 1.0)
    thr = cx.ThresholdTopK(0.01)
    cm[0].setThreshold(thr)
    cm[0].connectTx(1, 0)
    cm[1].connectRx(0, 0)
    torch.manual_seed(0)
    v = torch.randn(n, device=dev)
    cm[0].writeRemote(v)
    out = cm[1].readRemote()
    frac = float((out != 0).float().mean())
    assert 0.002 <= frac <= 0.03   # the estimate uses the 10th largest of 1000 samples: about top-k
    t = cm[0].threshold.getThreshold()
    assert torch.equal(out, torch.where(v.abs() > t, v, torch.zeros_like(v)))
    assert cm[0].getSize() == n


def test_comprex_variants_and_rests_api(world):
    n, dev = 4000, world.device
    cm = make(world, cx.Comprex, n, 3.0)
    cm[0].setThreshold(cx.ThresholdConst(1.0))
    cm[0].connectTx(1, 0)
    cm[1].connectRx(0, 0)
    torch.manual_seed(1)
    v = torch.randn(n, device=dev)
    big = v.abs() > 1.0
    cm[0].writeRemote_NoResidual(v)                      # the remainder is dropped
    assert torch.equal(cm[1].readRemote(), torch.where(big, v, torch.zeros_like(v)))
    assert float(cm[0].getRests().abs().sum()) == 0.0
    cm[0].writeRemote_compressOnly(v)                    # everything non-zero travels
    assert torch.equal(cm[1].readRemote(), v)
    cm[0].writeRemote(v)
    cm[1].readRemote()
    rest = cm[0].getRests()
    assert torch.equal(rest, torch.where(big, torch.zeros_like(v), v))
    x = torch.ones(n, device=dev)
    cm[0].addRests(x)
    assert torch.equal(x, 1 + rest)
    sd = cm[0].state_dict()
    cm[0].resetRests()
    assert float(cm[0].getRests().abs().sum()) == 0.0
    cm[0].load_state_dict(sd)
    assert torch.equal(cm[0].getRests(), rest)
    cm[0].setRests(np.zeros(n, dtype=np.float32))
    assert float(cm[0].getRests().abs().sum()) == 0.0
    with pytest.raises(cx.ComprexError, match="without connecting"):
        cm[2].writeRemote(v)
    with pytest.raises(cx.ComprexError, match="without connecting"):
        cm[2].readRemote()


def test_comprex_forwarding_ring(world):
    """0 -> 1 -> 2: rank 1 passes the compressed bytes on unchanged (readRemote_forward, forward_add)."""
    n, dev = 30000, world.device
    cm = make(world, cx.Comprex, n, 3.0, True)
    for c in cm:
        c.setThreshold(cx.ThresholdTopK(0.05))
    cm[0].connectTx(1, 0)
    cm[1].connectTo(0, 2, 0)
    cm[2].connectRx(1, 0)
    v = torch.randn(n, device=dev)
    cm[0].writeRemote(v)
    mid = torch.empty(n, device=dev)
    cm[1].readRemote_forward(mid)
    end = cm[2].readRemote()
    assert torch.equal(mid, end) and 0 < int((end != 0).sum()) < n // 5
    cm[0].writeRemote(v)
    acc = torch.ones(n, device=dev)
    cm[1].readRemote_wait()
    cm[1].forward_buffer()
    cm[1].forward_add(acc)
    end2 = cm[2].readRemote()
    assert torch.equal(acc, 1 + end2)


@pytest.mark.parametrize("codec", ["none", "rle"])
def test_comprex_other_codecs(world, codec):
    n, dev = 3000, world.device
    cm = make(world, cx.Comprex, n, 3.0)
    for c in cm:
        c.setCompressor(cx.CompressorNone() if codec == "none" else cx.CompressorRLE())
        c.setThreshold(cx.ThresholdConst(0.8))
    cm[0].connectTx(1, 0)
    cm[1].connectRx(0, 0)
    torch.manual_seed(2)
    v = torch.randn(n, device=dev)
    cm[0].writeRemote(v)
    out = cm[1].readRemote()
    if codec == "none":
        assert torch.equal(out, v)                       # dense payload: data + rests, rests = 0
    else:
        assert torch.equal(out, torch.where(v.abs() >= 0.8, v, torch.zeros_like(v)))
    acc = torch.ones(n, device=dev)
    cm[0].writeRemote(v)
    cm[1].readRemote_add(acc)
    total = out.clone()
    cm[0].flushRests()
    cm[1].readRemote_add(acc)
    assert torch.allclose(acc, 1 + 2 * v - total, atol=1e-6)


def test_fastcomprex_is_one_step_stale_and_conserves(world):
    n, dev = 20000, world.device
    fc = make(world, cx.FastComprex, n, 3.0)
    for c in fc:
        c.setThreshold(cx.ThresholdTopK(0.05))
    fc[0].connectTx(1, 0)
    fc[1].connectRx(0, 0)
    vals = alt_ramp(n, dev)
    acc = torch.zeros(n, device=dev)
    fc[0].writeRemote(vals)
    first = fc[1].readRemote()
    assert float(first.abs().sum()) == 0.0               # the first message is empty
    runs = 4
    for _ in range(runs - 1):
        fc[0].writeRemote(vals)
        fc[1].readRemote_add(acc)
    fc[0].flushRests()                                   # pending payload + residual
    fc[1].readRemote_add(acc)
    assert torch.equal(acc, runs * vals)
    # writeRemote_sameAs: a second engine sends the bytes the first one compressed
    a, b = make(world, cx.FastComprex, n, 3.0), make(world, cx.FastComprex, n, 3.0)
    for c in a + b:
        c.setThreshold(cx.ThresholdTopK(0.05))
    a[0].connectTx(1, 0)
    b[0].connectTx_sameBufferAs(2, 1, a[0])
    a[1].connectRx(0, 0)
    b[2].connectRx(0, 1)
    for _ in range(3):
        a[0].writeRemote(vals)
        b[0].writeRemote_sameAs(a[0])
        ra, rb = a[1].readRemote(), b[2].readRemote()
        assert torch.equal(ra, rb)
    assert float(ra.abs().sum()) > 0


@pytest.mark.gpu
@pytest.mark.parametrize("n", [5003, (1 << 24) + 3])
@pytest.mark.parametrize("kind", ["pairs", "exact", "rle", "dense"])
@pytest.mark.parametrize("add", [True, False])
def test_receive_into_the_vector_just_sent(n, kind, add):
    """writeRemote(v) and then a receive into the same v, while the peer's message is already there: the
    receive kernel has nothing to wait for but the sender in front of it, which must have read all of v."""
    world = cx.LoopbackWorld(2, device="cuda", timeout_ms=2000)
    ex = [cx.GaspiEx(e, n) if kind == "dense" else cx.Comprex(e, n) for e in world.envs]
    for r, e in enumerate(ex):
        if kind != "dense":
            e.setThreshold(cx.ThresholdTopK(0.1, exact=kind == "exact"))
            e.setCompressor(cx.CompressorRLE() if kind == "rle" else cx.CompressorIndexPairs())
        e.connectTo(1 - r, 1 - r)
    gen = torch.Generator(device="cuda").manual_seed(n)
    kept = [torch.zeros(n, device="cuda") for _ in ex]
    for _ in range(3):
        v, peer = (torch.randn(n, device="cuda", generator=gen) for _ in range(2))
        before = v.clone()
        torch.cuda.synchronize()
        ex[1].writeRemote(peer)
        ex[0].writeRemote(v)
        if add:
            ex[0].readRemote_add(v)
        else:
            (ex[0].readRemote_vec if kind == "dense" else ex[0].readRemote)(v)
        got = torch.empty(n, device="cuda")
        (ex[1].readRemote_vec if kind == "dense" else ex[1].readRemote)(got)
        if kind == "dense":
            sent, here = before, peer
        else:
            # an element is either sent or kept: both sums are exact
            sent = before + kept[0] - ex[0].getRests()
            here = peer + kept[1] - ex[1].getRests()
            kept = [e.getRests() for e in ex]
        assert torch.equal(got, sent) and torch.equal(v, before + here if add else here)
        for e in world.envs:
            e.check()
    world.close()


@pytest.mark.gpu
@pytest.mark.parametrize("how", ["exact", "exact_ties", "sample", "large_sample"])
@pytest.mark.parametrize("kind", ["pairs", "rle", "dense"])
def test_receive_behind_a_threshold_of_the_same_vector(how, kind):
    """writeRemote(x), a threshold of y, then a receive into y whose message is already there: the threshold
    kernels let the receive kernel in early, and may read y again after that (candidates that do not fit,
    a sample that exceeds one CTA)."""
    world = cx.LoopbackWorld(2, device="cuda", timeout_ms=2000)
    n = (1 << 22) + 3
    ex = [cx.GaspiEx(e, n) if kind == "dense" else cx.Comprex(e, n) for e in world.envs]
    for r, e in enumerate(ex):
        if kind != "dense":
            e.setThreshold(cx.ThresholdTopK(0.1))
            e.setCompressor(cx.CompressorRLE() if kind == "rle" else cx.CompressorIndexPairs())
        e.connectTo(1 - r, 1 - r)
    ratio = {"sample": 0.01, "large_sample": 0.0004}.get(how, 0.3)
    gen = torch.Generator(device="cuda").manual_seed(4)
    for _ in range(3):
        x, y, peer = (torch.randn(n, device="cuda", generator=gen) for _ in range(3))
        if how == "exact_ties":
            y = torch.randint(0, 4, (n,), device="cuda", generator=gen).float()
        if how.startswith("exact"):
            want = float(y.abs().sort(descending=True).values[math.ceil(np.float32(n) * np.float32(ratio)) - 1])
        else:
            want = ref_threshold_topk(y, ratio)
        before = y.clone()
        thr = cx.ThresholdTopK(ratio, exact=how.startswith("exact"))
        torch.cuda.synchronize()
        ex[1].writeRemote(peer)
        ex[0].writeRemote(x)
        thr.prepare(y)
        ex[0].readRemote_add(y)
        assert thr.getThreshold() == want
        here = peer
        if kind != "dense":
            here = peer - ex[1].getRests()
            ex[1].resetRests()
        assert torch.equal(y, before + here)
        (ex[1].readRemote_vec if kind == "dense" else ex[1].readRemote)(x)
        for e in world.envs:
            e.check()
    world.close()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["pairs", "dense"])
def test_two_threads_on_one_stream(kind):
    """Two threads, each with engines of its own, on the default stream: a receive kernel lets the next one in
    early, so the next receive into the same vector has to know that it is in front, whatever the other
    thread launches in between.  Whole numbers: all sums are exact."""
    n, rounds = (1 << 20) + 7, 60
    worlds = [cx.LoopbackWorld(2, device="cuda", timeout_ms=2000) for _ in range(2)]
    pairs = []
    for w in worlds:
        ex = [cx.GaspiEx(e, n) if kind == "dense" else cx.Comprex(e, n) for e in w.envs]
        for r, e in enumerate(ex):
            if kind != "dense":
                e.setThreshold(cx.ThresholdTopK(0.1))
                e.setCompressor(cx.CompressorIndexPairs())
            e.connectTo(1 - r, 1 - r)
        pairs.append(ex)
    out, err = [None, None], []

    def work(t):
        try:
            tx, rx = pairs[t]
            gen = torch.Generator(device="cuda").manual_seed(t)
            acc, total = torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
            for _ in range(rounds):
                for _ in range(2):
                    v = torch.randint(-9, 10, (n,), device="cuda", generator=gen).float()
                    total += v
                    tx.writeRemote(v)
                rx.readRemote_add(acc)
                rx.readRemote_add(acc)
            out[t] = (acc if kind == "dense" else acc + tx.getRests(), total)
        except BaseException as e:       # noqa: BLE001 - reported by the main thread
            err.append(e)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(2)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not err, err
    for got, want in out:
        assert torch.equal(got, want)
    for w in worlds:
        for e in w.envs:
            e.check()
        w.close()


@pytest.mark.gpu
@pytest.mark.parametrize("cls", ["Comprex", "GaspiEx"])
def test_unusual_vectors_raise(cls):
    """Vectors that have no address (sparse, wrapped by a transform) raise and leave the connection usable."""
    env = cx.GaspiEnvironment(1 << 20, device="cuda")
    n = 100
    ex = getattr(cx, cls)(env, n)
    if cls == "Comprex":
        ex.setThreshold(cx.ThresholdTopK(1.0))
        ex.setCompressor(cx.CompressorIndexPairs())
    ex.connectTo(0, 0)
    sparse = torch.sparse_coo_tensor([[1]], [1.0], (n,), device="cuda", check_invariants=True)
    for call in (ex.writeRemote, ex.readRemote_add):
        with pytest.raises(Exception):
            call(sparse)
        with pytest.raises(Exception):
            torch.func.vmap(lambda x: call(x) or x)(torch.zeros(3, n, device="cuda"))
    v, out = torch.randn(n, device="cuda"), torch.zeros(n, device="cuda")
    ex.writeRemote(v)
    ex.readRemote_add(out)
    assert torch.equal(out + (ex.getRests() if cls == "Comprex" else 0), v)
    env.check()
    env.close()


@pytest.mark.gpu
@pytest.mark.parametrize("cls", ["Comprex", "GaspiEx"])
def test_time_budget_changed_between_reads(cls):
    """A read waits as long as the environment says when it is issued, also behind earlier reads."""
    env = cx.GaspiEnvironment(1 << 20, device="cuda", timeout_ms=8000)
    n = 100
    ex = getattr(cx, cls)(env, n)
    if cls == "Comprex":
        ex.setThreshold(cx.ThresholdTopK(1.0))
        ex.setCompressor(cx.CompressorIndexPairs())
    ex.connectTo(0, 0)
    out = torch.zeros(n, device="cuda")
    for _ in range(4):
        ex.writeRemote(torch.ones(n, device="cuda"))
        ex.readRemote_add(out)
    env.flush()
    env.check()
    env.timeout_ns = 50_000_000
    start = time.perf_counter()
    ex.readRemote_add(out)                   # nothing was sent
    torch.cuda.synchronize()
    assert time.perf_counter() - start < 4.0
    with pytest.raises(cx.ComprexError, match="TIMEOUT"):
        env.check()
    env.close()


@pytest.mark.gpu
def test_prepared_sends_survive_a_change_to_exact_and_back():
    """A fraction so small that every element is sampled uses the small scratch; one message with exact top-k in
    between brings a larger one.  The launch list that was prepared before must not use memory that has
    become somebody else's."""
    env = cx.GaspiEnvironment(1 << 20, device="cuda")
    n = 30000
    ex = cx.Comprex(env, n)
    ex.setCompressor(cx.CompressorIndexPairs())
    ex.connectTo(0, 0)
    gen = torch.Generator(device="cuda").manual_seed(2)
    out, total, others = torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda"), []
    for k, exact in enumerate((False, False, True, False, False, False)):
        ex.setThreshold(cx.ThresholdTopK(1e-4, exact=exact))
        v = torch.randint(-1000, 1000, (n,), device="cuda", generator=gen).float()
        held = ex.getRests() + v
        want = held.abs().sort(descending=True).values[2]      # ceil(n * 1e-4) - 1
        total += v
        ex.writeRemote(v)
        ex.readRemote_add(out)
        assert ex.threshold.getThreshold() == float(want)
        assert torch.equal(out + ex.getRests(), total)
        others += [torch.full((1024,), 7, dtype=torch.int32, device="cuda") for _ in range(32)]
        assert all(bool((t == 7).all()) for t in others), k
    env.check()
    env.close()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["pairs", "rle", "dense"])
@pytest.mark.parametrize("read", ["add", "set"])
@pytest.mark.parametrize("side", [64, 256, 1024])
def test_program_work_between_send_and_receive(kind, read, side):
    """A matrix product of the program's own writes the receiver's vector between the two halves of a message: the
    receive kernel may be resident early, but touches the vector only behind that."""
    n = side * side
    env = cx.GaspiEnvironment(1 << 20, device="cuda")
    ex = cx.GaspiEx(env, n) if kind == "dense" else cx.Comprex(env, n)
    if kind != "dense":
        ex.setThreshold(cx.ThresholdTopK(0.05))
        ex.setCompressor(cx.CompressorRLE() if kind == "rle" else cx.CompressorIndexPairs())
    ex.connectTo(0, 0)
    gen = torch.Generator(device="cuda").manual_seed(side)
    out, held = torch.empty(n, device="cuda"), torch.zeros(n, device="cuda")
    for _ in range(8):
        v = torch.randint(-9, 10, (n,), device="cuda", generator=gen).float()
        a, b = (torch.randint(-2, 3, (side, side), device="cuda", generator=gen).float() for _ in range(2))
        product = (a @ b).view(n)
        out.fill_(1e6)
        ex.writeRemote(v)
        torch.mm(a, b, out=out.view(side, side))
        if read == "add":
            ex.readRemote_add(out)
        elif kind == "dense":
            ex.readRemote_vec(out, n)
        else:
            ex.readRemote(out)
        held += v
        if kind != "dense":
            sent, held = held - ex.getRests(), ex.getRests()
        else:
            sent = v
        assert torch.equal(out, (product if read == "add" else 0) + sent)
    env.check()
    env.close()


@pytest.mark.parametrize("codec_first", [False, True])
def test_run_length_scratch_comes_with_the_sending_side(world, codec_first):
    """The sender's workspace (4.1 bytes an element) is made when an engine connects to send, in either order with
    the codec; an engine that only receives has none, and messages arrive whatever the memory held before."""
    n, dev = 70001, world.device
    junk = [torch.full((n,), 7, dtype=torch.int32, device=dev) for _ in range(8)]
    del junk
    ex = make(world, cx.Comprex, n)
    for e in ex:
        e.setThreshold(cx.ThresholdTopK(0.1))
    if not codec_first:
        ex[0].connectTx(1)
        ex[1].connectRx(0)
    for e in ex:
        e.setCompressor(cx.CompressorRLE())
    if codec_first:
        ex[0].connectTx(1)
        ex[1].connectRx(0)
    assert ex[0]._rle.tx_ws is not None and ex[1]._rle.tx_ws is None and ex[2]._rle.tx_ws is None
    held = torch.zeros(n, device=dev)
    for _ in range(3):
        v = torch.randint(-50, 50, (n,), device=dev).float()
        ex[0].writeRemote(v)
        out = torch.ones(n, device=dev)
        ex[1].readRemote_add(out)
        held += v
        assert torch.equal(out - 1 + ex[0].getRests(), held)
        held = ex[0].getRests()
    assert ex[1]._rle.tx_ws is None
