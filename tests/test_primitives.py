"""Unit tests of the native primitives against plain PyTorch fp32 restatements.

Every test runs on the host implementation (CPU) and, marked ``gpu``, on the
CUDA kernels; the CUDA kernels are additionally compared bit for bit with the
host implementation of the same primitive.
"""
import ctypes as C

import pytest
import torch

import comprex_b200 as cx
from comprex_b200 import _lib
from comprex_b200.ops import primitives as P

from helpers import ref_compress, ref_threshold_topk

SIZES = [1, 31, 32, 33, 1023, 1024, 1025, 4095, 4096, 4097, 10007, 70001]


@pytest.fixture
def world(device):
    w = cx.LoopbackWorld(2, device=device, timeout_ms=200)
    yield w
    w.close()


def read_pairs(env, slot, rank=None):
    """Header, pairs in index order, and the per-sub-tile counts of a slot.

    Sub-tiles sit in the pair list in the order of their reservations; the table entry
    {start, count} of each sub-tile must address exactly its own pairs, each index once.
    """
    ep = slot.endpoint(env, rank)
    hdr = env.read_header(ep.hdr)
    raw = env.read_bytes(ep.pairs, 8 * slot.cap)    # the list may have gaps between its regions
    buf = torch.frombuffer(bytearray(raw), dtype=torch.int32).view(-1, 2)
    nsub = (hdr.n + _lib.SUBTILE - 1) // _lib.SUBTILE
    traw = env.read_bytes(ep.table, 8 * max(nsub, 1))[: 8 * nsub]
    table = torch.frombuffer(bytearray(traw), dtype=torch.int32).view(-1, 2).clone() if nsub else torch.zeros(0, 2, dtype=torch.int32)
    idx_parts, val_parts = [], []
    for s_ in range(nsub):
        start, count = int(table[s_, 0]), int(table[s_, 1])
        assert start + count <= slot.cap
        part = buf[start:start + count]
        i = part[:, 0]
        assert bool((i >= s_ * _lib.SUBTILE).all()) and bool((i < (s_ + 1) * _lib.SUBTILE).all())
        order = torch.argsort(i)                  # the order inside a sub-tile is not part of the format
        i = i[order]
        assert bool((i[1:] > i[:-1]).all())      # but every index occurs once
        idx_parts.append(i.clone())
        val_parts.append(part[:, 1][order].clone().view(torch.float32))
    idx = torch.cat(idx_parts) if idx_parts else torch.zeros(0, dtype=torch.int32)
    val = torch.cat(val_parts) if val_parts else torch.zeros(0)
    assert idx.numel() == hdr.nnz            # every stored pair belongs to exactly one sub-tile
    return hdr, idx, val, table[:, 1].clone()


@pytest.mark.parametrize("n", [1, 50, 999, 1000, 1001, 4096, 100003, 1 << 20])
@pytest.mark.parametrize("ratio", [0.1, 0.01, 0.001])
def test_threshold_matches_reference_rule(device, n, ratio):
    torch.manual_seed(n)
    env = cx.GaspiEnvironment(1 << 16, device=device)
    g = torch.randn(n).to(device)
    r = (0.5 * torch.randn(n)).to(device)
    comp = P.Compressor(env, n)
    comp.threshold_topk(g, r, n, ratio)
    got = comp.thr.item()
    want = ref_threshold_topk(r.cpu() + g.cpu(), ratio)
    assert got == want
    # sampling parameters of the ring variants
    comp.threshold_topk(g, None, n, ratio, 250, 4.0)
    assert comp.thr.item() == ref_threshold_topk(g.cpu(), ratio, 250, 4.0)
    env.close()


@pytest.mark.parametrize("n,ratio", [(999, 0.05), (30000, 0.01), (150001, 0.002)])
def test_exact_topk_threshold(device, n, ratio):
    """exact=True: the threshold is the ceil(n*ratio)-th largest magnitude of the whole vector
    (for n above the shared-memory key cache the kernel re-reads the vector in every pass)."""
    torch.manual_seed(n)
    env = cx.GaspiEnvironment(1 << 16, device=device)
    g, r = torch.randn(n).to(device), (0.3 * torch.randn(n)).to(device)
    thr = cx.ThresholdTopK(ratio, exact=True)
    thr.prepare_with(r, g)
    mags = (g + r).abs().cpu().sort(descending=True).values
    k = int(torch.ceil(torch.tensor(float(n) * ratio)).item())
    assert thr.getThreshold() == float(mags[k - 1])
    comp = P.Compressor(env, n)
    thr._launch(comp, g, r, n)
    assert comp.thr.item() == float(mags[k - 1])
    assert int(((g + r).abs() > comp.thr).sum()) == k - 1      # strict ">" of the pair codec
    env.close()


@pytest.mark.gpu
@pytest.mark.parametrize("data", ["normal", "columns", "ties", "few_values", "zeros", "constant", "nan"])
@pytest.mark.parametrize("n,dtype", [(11009, torch.float32), (65536, torch.bfloat16), (1000003, torch.float32),
                                     (1 << 21, torch.float16)])
def test_exact_topk_one_pass(n, dtype, data):
    """The one-pass exact selection (bracket from a sample, candidates, finish) equals a sort for all
    ranks, where the bracket holds, where its ends are ties, and where the candidates do not fit and
    it selects over the whole vector; the scratch is left clean."""
    gen = torch.Generator(device="cuda").manual_seed(n)
    g = torch.randn(n, device="cuda", generator=gen)
    if data == "columns":                      # every 1024th element is large
        g[::1024] *= 1000.0
    elif data == "ties":
        g = g.mul(2.0).round()
    elif data == "few_values":
        g = torch.randint(0, 4, (n,), device="cuda", generator=gen).float() * 0.125 + 1.0
    elif data == "zeros":
        g[torch.rand(n, device="cuda", generator=gen) < 0.999] = 0.0
    elif data == "constant":
        g.fill_(-3.0)
    elif data == "nan":
        g[5] = float("nan")
    g = g.to(dtype)
    r = torch.zeros(n, device="cuda") if data == "few_values" else torch.full((n,), 0.25, device="cuda")
    keys = (r + g.float()).abs().view(torch.int32).sort(descending=True).values
    env = cx.GaspiEnvironment(1 << 16, device="cuda")
    comp = P.Compressor(env, n)
    for ratio in (0.0005, 0.01, 0.1, 0.5, 1.0):
        k = int(torch.ceil(torch.tensor(float(n)) * torch.tensor(ratio)).item()) - 1
        if k <= 0:
            continue
        for _ in range(2):
            comp.threshold_topk(g, r, n, ratio, cx.ThresholdTopK.EXACT)
            assert int(comp.thr.view(torch.int32).item()) == int(keys[k].item()), (ratio, k)
    env.close()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_exact_topk_candidates_in_few_ctas(dtype):
    """The elements around the wanted rank lie where the same few CTAs come by, round after round: their
    buffers fill up, are emptied between rounds, and what they have no room for goes to the list at once."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for per_sm in (4, 5, 6):                   # resident CTAs of the collecting kernel
        grid, chunk, rounds = sms * per_sm, 2048, 20
        n = grid * chunk * rounds
        gen = torch.Generator(device="cuda").manual_seed(per_sm)
        values = (0.5 + torch.rand(n, device="cuda", generator=gen)).to(dtype).float().sort().values
        hot = max(1, round(0.04 * grid))       # CTAs that meet the middle 4 % of the values
        mid0 = n // 2 - hot * rounds * chunk // 2
        mid, rest = values[mid0:mid0 + hot * rounds * chunk], torch.cat((values[:mid0], values[mid0 + hot * rounds * chunk:]))
        g = torch.empty(rounds, grid, chunk, device="cuda")
        g[:, :hot] = mid.view(rounds, hot, chunk)
        g[:, hot:] = rest[torch.randperm(rest.numel(), device="cuda", generator=gen)].view(rounds, grid - hot, chunk)
        env = cx.GaspiEnvironment(1 << 16, device="cuda")
        comp = P.Compressor(env, n)
        comp.threshold_topk(g.view(-1).to(dtype), None, n, 0.5, cx.ThresholdTopK.EXACT)
        k = int(torch.ceil(torch.tensor(float(n)) * torch.tensor(0.5)).item()) - 1
        assert float(comp.thr) == float(values[n - 1 - k])
        env.close()


@pytest.mark.gpu
@pytest.mark.parametrize("count", [0, 1, 31, 128, 129, 255, 256, 257, 1024])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shift", [0, 1])
def test_set_of_one_source(count, dtype, shift):
    """Sub-tiles on both sides of the count up to which values go straight to their places, a partial one at
    the end, and a destination that takes no wide accesses: every other element is overwritten with zero."""
    n = 3 * 1024 + 500
    world = cx.LoopbackWorld(1, device="cuda", timeout_ms=2000)
    e0 = world.envs[0]
    gen = torch.Generator().manual_seed(count)
    keep = torch.zeros(n, dtype=torch.bool)
    for sub in range(0, n, 1024):
        room = min(1024, n - sub)
        keep[sub + torch.randperm(room, generator=gen)[:count]] = True
    x = torch.where(keep, torch.randn(n, generator=gen).abs() + 0.5, torch.zeros(n))
    comp, slot = P.Compressor(e0, n), P.SparseSlot.create(e0, n, n)
    comp.set_threshold(0.25)
    comp.compress(x.cuda(), None, n, n, 1, P.make_targets([slot.endpoint(e0)]))
    out = torch.full((n + 1,), 9.0, dtype=dtype, device="cuda")
    status = e0.new_status("t")
    P.apply_sparse(e0, P.make_sources([slot.endpoint(e0)], [1]), n, P.args_set(out[shift:shift + n], 0.5), status)
    e0.flush()
    assert status.value == 0
    assert torch.equal(out[shift:shift + n].cpu(), (0.5 * x).to(dtype))
    assert float(out[n if shift == 0 else 0]) == 9.0
    world.close()


@pytest.mark.gpu
@pytest.mark.parametrize("subs,count", [(3, c) for c in (101, 102, 103)] + [(8000, c) for c in (0, 14, 15, 16, 129, 1024)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shift", [0, 1])
def test_set_of_one_source_by_length(subs, count, dtype, shift):
    """Sub-tiles on both sides of the counts up to which values go straight to their places, in a vector of one
    sub-tile per warp and in a longer one, a partial one at the end, and a destination that takes no wide
    accesses: every other element is overwritten with zero."""
    n = subs * 1024 + 500
    world = cx.LoopbackWorld(1, device="cuda", timeout_ms=2000)
    e0 = world.envs[0]
    gen = torch.Generator().manual_seed(count)
    keep = torch.zeros(n, dtype=torch.bool)
    place = torch.randperm(1024, generator=gen)          # every sub-tile's places are the one's before, moved on
    for sub in range(0, n, 1024):
        at = (place + 7 * (sub // 1024)) % 1024
        keep[sub + at[at < n - sub][:count]] = True
    x = torch.where(keep, torch.randn(n, generator=gen).abs() + 0.5, torch.zeros(n))
    cap = n + 32 * 1024                        # every region has room for its sub-tiles
    comp, slot = P.Compressor(e0, n), P.SparseSlot.create(e0, n, cap)
    comp.set_threshold(0.25)
    comp.compress(x.cuda(), None, n, cap, 1, P.make_targets([slot.endpoint(e0)]))
    out = torch.full((n + 1,), 9.0, dtype=dtype, device="cuda")
    status = e0.new_status("t")
    P.apply_sparse(e0, P.make_sources([slot.endpoint(e0)], [1]), n, P.args_set(out[shift:shift + n], 0.5), status)
    e0.flush()
    assert status.value == 0
    assert torch.equal(out[shift:shift + n].cpu(), (0.5 * x).to(dtype))
    assert float(out[n if shift == 0 else 0]) == 9.0
    world.close()


@pytest.mark.gpu
@pytest.mark.parametrize("data", ["normal", "ties", "constant", "ends"])
@pytest.mark.parametrize("n", [33, 1000, 1024, 1025, 2049, 11008])
def test_threshold_selection_ranks(n, data):
    """Both selections at the edges of their ranges: ranks around 32 and 768, samples around 1024 (the kernel for up
    to 2048 samples) and at the cluster's first and last size, few distinct keys."""
    torch.manual_seed(n)
    g = torch.randn(n)
    if data == "ties":
        g = g.mul(2.0).round()
    elif data == "constant":
        g.fill_(-3.0)
    elif data == "ends":                       # only zeros and infinities
        g = torch.where(g > 0.5, torch.inf, 0.0)
    keys = g.abs().sort(descending=True).values
    env = cx.GaspiEnvironment(1 << 16, device="cuda")
    comp, dev = P.Compressor(env, n), g.cuda()
    for rank in (1, 9, 31, 32, 99, 767, 768, n // 2, n - 1):
        ratio = (rank + 0.5) / n               # ceil(n * ratio) - 1 == rank
        if rank < n and ratio < 1.0:
            comp.threshold_topk(dev, None, n, ratio, n, 1.0)
            assert comp.thr.item() == float(keys[rank]), rank
    env.close()


@pytest.mark.gpu
@pytest.mark.parametrize("large", [0, 12000, 30000])
@pytest.mark.parametrize("data", ["normal", "ties"])
def test_thresholds_that_share_a_launch(large, data):
    """Several vectors in one list: samples of up to 2048 alone, and beside one that is larger than the cluster's
    (they then take the large kernel, with every rank): each the reference's value."""
    env = cx.GaspiEnvironment(1 << 16, device="cuda")
    gen = torch.Generator().manual_seed(large)
    todo = [(5, 0.5, 1000), (700, 0.1, 1000), (1000, 0.9, 1024), (1024, 0.01, 1024), (2048, 0.3, 2048), (3000, 0.02, 1500)]
    if large:
        todo.insert(3, (large + 17, 0.01, large))
    ops, keep = (_lib.Op * len(todo))(), []
    for o, (n, ratio, samples) in zip(ops, todo):
        x = torch.randn(n, generator=gen)
        if data == "ties":
            x = x.mul(2.0).round()
        comp, dev = P.Compressor(env, n), x.cuda()
        o.kind, o.dev, o.n, o.dtype, o.g, o.thr = _lib.OPK_THRESHOLD, env.dev, n, _lib.F32, dev.data_ptr(), comp.thr.data_ptr()
        o.ratio, o.default_subsamples, o.subsample_factor = ratio, samples, 0.0
        keep.append((comp, dev, x))
    _lib.check(env.lib.cx_run_ops(ops, len(todo), 1, _lib.stream_ptr(env.device)))
    env.flush()
    for (comp, _, x), (n, ratio, samples) in zip(keep, todo):
        assert float(comp.thr) == ref_threshold_topk(x, ratio, samples, 0.0), (n, ratio)
    env.close()


def test_threshold_reference_vector(device):
    """test/threshold.cpp:58-85: 100 ints, top 10 % -> threshold 90, 10 elements pass with >=."""
    from helpers import alt_ramp
    v = alt_ramp(100, device)
    thr = cx.ThresholdTopK(0.10)
    thr.prepare(v)
    assert thr.getThreshold() == 90.0
    kept = thr.apply(v)
    assert int((kept != 0).sum()) == 10
    const = cx.ThresholdConst(20)
    assert int((const.apply(v) != 0).sum()) == 80


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_compress_add_update(world, n, dtype):
    torch.manual_seed(n)
    e0, e1 = world.envs
    dev = world.device
    cap = n
    slot0 = P.SparseSlot.create(e0, n, cap)
    slot1 = P.SparseSlot.create(e1, n, cap)
    assert slot0.alloc == slot1.alloc
    g = torch.randn(n).to(dtype).to(dev)
    r0 = (0.3 * torch.randn(n)).to(dev)
    r = r0.clone()
    comp = P.Compressor(e0, n)
    comp.set_threshold(1.0)
    comp.compress(g, r, n, cap, 7, P.make_targets([slot1.endpoint(e0, 1), slot0.endpoint(e0, 0)]))
    e0.flush()
    idx_w, val_w, r_w = ref_compress(g.cpu(), r0.cpu(), 1.0)
    for env, slot in ((e1, slot1), (e0, slot0)):
        hdr, idx, val, prefix = read_pairs(env, slot)
        assert hdr.seq == 7 and hdr.n == n and hdr.kind == _lib.KIND_PAIRS
        assert hdr.nnz == idx_w.numel() == hdr.nnz_found
        assert torch.equal(idx, idx_w)           # the same set of survivors as the reference codec
        assert torch.equal(val, val_w)
        # counts[s] == number of survivors with index in [s*1024, (s+1)*1024)
        want = torch.bincount(idx_w.long() // _lib.SUBTILE, minlength=prefix.numel())
        assert torch.equal(prefix.long(), want)
    assert torch.equal(r.cpu(), r_w)
    # conservation: what was sent plus what stayed equals what came in
    dense = torch.zeros(n)
    dense[idx_w.long()] = val_w
    assert torch.equal(dense + r.cpu(), r0.cpu() + g.cpu().float())
    st = comp.last_stats()
    assert st["nnz"] == idx_w.numel() and st["status"] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1024, 4097, 70001, (1 << 20) + 5])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("mode", ["add_update", "update", "plain"])
def test_compress_bulk_copy_kernel_matches_register_kernel(monkeypatch, n, dtype, mode):
    """The opt-in compress kernel whose sub-tiles arrive through bulk copies into shared memory
    (cp.async.bulk + mbarrier, a pipeline per warp) selects the same survivors, writes the same
    table counts and leaves the same residual as the default kernel, for all three modes, on
    sizes with a partial last sub-tile, and with a slot that overflows."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    results = []
    for bulk in ("0", "1"):
        monkeypatch.setenv("COMPREX_COMPRESS_BULK", bulk)
        world = cx.LoopbackWorld(2, device="cuda", timeout_ms=2000)
        e0, e1 = world.envs
        gen = torch.Generator().manual_seed(n)
        g = torch.randn(n, generator=gen).to(dtype).cuda()
        r = (0.3 * torch.randn(n, generator=gen)).cuda()
        out = []

        def run(cap, rr, seq, slot, comp):
            tg = P.make_targets([slot.endpoint(e0, 1)])
            if mode == "add_update":
                comp.compress(g, rr, n, cap, seq, tg)
            elif mode == "update":
                comp.compress(None, rr, n, cap, seq, tg)
            else:
                comp.compress(g, None, n, cap, seq, tg)
            e0.flush()
            hdr, idx, val, counts = read_pairs(e1, slot)
            return hdr, idx, val, counts, comp.last_stats()

        P.SparseSlot.create(e0, n, n)                 # allocations are symmetric across the ranks
        slot = P.SparseSlot.create(e1, n, n)
        comp = P.Compressor(e0, n)
        comp.set_threshold(1.0)
        for seq in (1, 2):
            hdr, idx, val, counts, st = run(n, r, seq, slot, comp)
            assert hdr.nnz == hdr.nnz_found and st["status"] == 0
            out.append((hdr.nnz, idx, val, counts, r.cpu().clone()))
            r.add_(0.5)                               # something to send in the second round
        # a slot that overflows: which sub-tiles find room is a matter of timing, the totals are not
        cap = max(n // 64, 8)
        P.SparseSlot.create(e0, n, cap)
        slot = P.SparseSlot.create(e1, n, cap)
        hdr, idx, val, counts, st = run(cap, r.clone(), 1, slot, comp)
        assert hdr.nnz < hdr.nnz_found and st["status"] & _lib.ST_OVERFLOW
        out.append((hdr.nnz, hdr.nnz_found))
        results.append(out)
        world.close()
    for a, b in zip(*results):
        assert len(a) == len(b)
        for x, y in zip(a, b):
            assert torch.equal(x, y) if isinstance(x, torch.Tensor) else x == y


def test_compress_capacity_overflow_keeps_residual(world):
    e0, e1 = world.envs
    dev, n, cap = world.device, 20000, 100
    slot = [P.SparseSlot.create(e, n, cap) for e in world.envs][1]
    g = torch.randn(n).to(dev)
    r = torch.zeros(n, device=dev)
    comp = P.Compressor(e0, n)
    comp.set_threshold(0.5)
    comp.compress(g, r, n, cap, 1, P.make_targets([slot.endpoint(e0, 1)]))
    hdr, idx, val, _ = read_pairs(e1, slot)
    assert hdr.nnz == cap and hdr.nnz_found == int((g.abs() > 0.5).sum())
    # which survivors made it depends on the order of the reservations; whatever was
    # emitted passed the threshold and left the residual, everything else stayed in it
    sent = torch.zeros(n)
    sent[idx.long()] = val
    assert bool((val.abs() > 0.5).all()) and idx.unique().numel() == cap
    assert torch.equal(sent + r.cpu(), g.cpu())
    assert float((r.cpu()[idx.long()]).abs().sum()) == 0.0
    assert comp.last_stats()["status"] & _lib.ST_OVERFLOW
    e0.check()  # overflow is soft: no exception


@pytest.mark.gpu
@pytest.mark.parametrize("share", [2, 64])
@pytest.mark.parametrize("has_g", [False, True])
def test_compress_overflow_in_every_cta(share, has_g):
    """A dense vector through a slot of n / share pairs: the survivors of every CTA of a full grid do not
    fit.  The payload is published all the same, every region is full, and what was not sent stays."""
    world = cx.LoopbackWorld(2, device="cuda", timeout_ms=2000)
    e0, e1 = world.envs
    n = (1 << 24) + 5
    cap = n // share
    slot = [P.SparseSlot.create(e, n, cap) for e in world.envs][1]
    gen = torch.Generator(device="cuda").manual_seed(share)
    r = torch.randn(n, device="cuda", generator=gen).abs_().add_(0.25)
    g = torch.randn(n, device="cuda", generator=gen).abs_() if has_g else None
    x = r + g if has_g else r.clone()
    comp = P.Compressor(e0, n)
    comp.set_threshold(0.0)
    comp.compress(g, r, n, cap, 1, P.make_targets([slot.endpoint(e0, 1)]))
    e0.flush()
    st = comp.last_stats()
    assert st["status"] == _lib.ST_OVERFLOW
    regions, region_size = P.compress_regions(n, cap)
    hdr, idx, val, _ = read_pairs(e1, slot)
    assert hdr.seq == 1 and hdr.nnz_found == n and hdr.nnz == st["nnz"] == regions * region_size
    sent = torch.zeros(n)
    sent[idx.long()] = val
    assert idx.unique().numel() == hdr.nnz and torch.equal(sent + r.cpu(), x.cpu())
    world.close()


@pytest.mark.parametrize("mode", ["update", "plain"])
def test_compress_modes(world, mode):
    e0, e1 = world.envs
    dev, n = world.device, 5000
    slot = [P.SparseSlot.create(e, n, n) for e in world.envs][1]
    x = torch.randn(n).to(dev)
    x[::3] = 0
    comp = P.Compressor(e0, n)
    comp.set_threshold(0.0)
    if mode == "update":   # flushRests: everything non-zero leaves, the residual ends up zero
        r = x.clone()
        comp.compress(None, r, n, n, 1, P.make_targets([slot.endpoint(e0, 1)]))
        assert int(r.abs().sum().item()) == 0
    else:                  # compressOnly: the input is untouched
        comp.compress(x, None, n, n, 1, P.make_targets([slot.endpoint(e0, 1)]))
    hdr, idx, val, _ = read_pairs(e1, slot)
    nz = torch.nonzero(x.cpu()).flatten()
    assert torch.equal(idx.long(), nz) and torch.equal(val, x.cpu()[nz])


def _fill_slots(world, n, nsrc, seed=0):
    """Each virtual rank j < nsrc compresses its own vector into rank 0's slot j."""
    torch.manual_seed(seed)
    dev = world.device
    e0 = world.envs[0]
    slots = [[P.SparseSlot.create(e, n, n) for e in world.envs] for _ in range(nsrc)]
    dense = []
    for j in range(nsrc):
        x = torch.randn(n)
        x[torch.rand(n) > 0.2] = 0
        dense.append(x)
        comp = P.Compressor(e0, n)
        comp.set_threshold(0.0)
        comp.compress(x.to(dev), None, n, n, 3, P.make_targets([slots[j][0].endpoint(e0, 0)]))
    src = P.make_sources([slots[j][0].endpoint(e0, 0) for j in range(nsrc)], [3] * nsrc)
    return src, dense


@pytest.mark.parametrize("n", [1, 1000, 1024, 4097, 50001])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_apply_add_and_set(world, n, out_dtype):
    e0 = world.envs[0]
    dev = world.device
    src, dense = _fill_slots(world, n, 3)
    st = e0.new_status("t")
    base = torch.randn(n).to(out_dtype)
    out = base.clone().to(dev)
    P.apply_sparse(e0, src, n, P.args_add(out, 0.5), st)
    want = base.clone()
    for d in dense:   # same order, same rounding as the kernel: one source after the other
        want = (want.float() + 0.5 * d).to(out_dtype)
    assert torch.equal(out.cpu(), want)
    out2 = torch.full((n,), 7.0, dtype=out_dtype, device=dev)
    P.apply_sparse(e0, src, n, P.args_set(out2, 0.25), st)
    acc = torch.zeros(n)
    for d in dense:
        acc += d
    assert torch.equal(out2.cpu(), (0.25 * acc).to(out_dtype))
    e0.flush()
    assert st.value == 0


@pytest.mark.parametrize("counts", [[0], [1024], [0, 0, 33], [31, 32, 33, 0, 1, 1024, 0, 64, 65, 0], [257] * 3 + [0] * 9])
def test_apply_set_segment_lengths(world, counts):
    """Segments of a sub-tile at the edges of the decode's rows of 32 pairs and batches of rows."""
    e0, dev, n = world.envs[0], world.device, 3 * 1024 + 100
    torch.manual_seed(len(counts))
    eps, want = [], torch.zeros(n)
    for c in counts:
        x = torch.zeros(n)
        for k, base in enumerate((0, 1024, 2048, 3072)):     # the second sub-tile is full, the third empty
            tile = min(1024, n - base)
            m = min(tile, (c, 1024 if c else 0, 0, c)[k])
            x[base + torch.randperm(tile)[:m]] = torch.randn(m)
        slot = P.SparseSlot.create(e0, n, n)
        for e in world.envs[1:]:
            P.SparseSlot.create(e, n, n)
        comp = P.Compressor(e0, n)
        comp.set_threshold(0.0)
        comp.compress(x.to(dev), None, n, n, 3, P.make_targets([slot.endpoint(e0, 0)]))
        eps.append(slot.endpoint(e0, 0))
        want += x
    st, out = e0.new_status("t"), torch.full((n,), 7.0, device=dev)
    P.apply_sparse(e0, P.make_sources(eps, [3] * len(eps)), n, P.args_set(out, 1.0), st)
    e0.flush()
    assert st.value == 0 and torch.equal(out.cpu(), want)


@pytest.mark.gpu
@pytest.mark.parametrize("op", ["add", "sgd"])
def test_apply_sparse_large_groups(op):
    """Vectors so long that a warp of the sparse decode takes 16 sub-tiles or more at a time."""
    env = cx.GaspiEnvironment(1 << 16, device="cuda")
    n = (1 << 27) + 5
    gen = torch.Generator(device="cuda").manual_seed(3)
    x = torch.zeros(n, device="cuda")
    at = torch.randint(0, n, (1 << 20,), device="cuda", generator=gen)
    x[at] = torch.randn(at.numel(), device="cuda", generator=gen)
    x[5 * 1024:7 * 1024] = 1.5                     # two full sub-tiles
    cap = 1 << 21
    slot, comp, st = P.SparseSlot.create(env, n, cap), P.Compressor(env, n), env.new_status("t")
    comp.set_threshold(0.0)
    comp.compress(x, None, n, cap, 3, P.make_targets([slot.endpoint(env, 0)]))
    src = P.make_sources([slot.endpoint(env, 0)], [3])
    out = torch.ones(n, device="cuda")
    args = P.args_add(out, 0.5) if op == "add" else P.args_update(_lib.OP_SGD, out, 0.25)
    P.apply_sparse(env, src, n, args, st)
    env.flush()
    assert st.value == 0 and torch.equal(out, 1 + 0.5 * x if op == "add" else 1 - 0.25 * x)
    env.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1000, 70001, 148 * 48 * 1024, 148 * 48 * 3 * 1024 + 1, 148 * 48 * 3 * 1024 + 1025, 50_000_003])
@pytest.mark.parametrize("nsrc", [2, 7, 15])
@pytest.mark.parametrize("density", [0.0005, 0.01, 0.2])
@pytest.mark.parametrize("what", ["add", "add_bf16", "sgd_shadow"])
def test_apply_sparse_several_sources(n, nsrc, density, what):
    """The sparse decode of several sources at the edges of its walks (batches of 128 pairs per sub-tile, groups
    of sub-tiles by the sources' pair counts): every element takes the sources one after the other, rounded
    after each; elements that several sources address, sub-tiles that are full in all of them, empty ones."""
    if n > 10_000_000 and (nsrc == 15 or (nsrc == 2 and what != "add")):
        pytest.skip("large vectors with seven sources, and with two where the result is fp32")
    env = cx.GaspiEnvironment(1 << 16, device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(nsrc)
    dt = torch.bfloat16 if what == "add_bf16" else torch.float32
    out = torch.randn(n, device="cuda", generator=gen).to(dt)
    shadow = torch.zeros(n, dtype=torch.bfloat16, device="cuda") if what == "sgd_shadow" else None
    want = out.clone()
    slots, st = [], env.new_status("t")
    touched = torch.zeros(n, dtype=torch.bool, device="cuda")
    for j in range(nsrc):
        x = torch.randn(n, device="cuda", generator=gen)
        x[torch.rand(n, device="cuda", generator=gen) >= density] = 0
        x[: min(n, 40)] = 1.0 + j                                    # elements of every source
        if n > 8192:
            x[2048:3072] = 0.5 + j                                   # a full sub-tile
            x[4096:5120] = 0
        cap = 32 * ((int((x != 0).sum()) // 16) + 1024 + 256)        # regions fill unevenly
        slot, comp = P.SparseSlot.create(env, n, cap), P.Compressor(env, n)
        comp.set_threshold(0.0)
        comp.compress(x, None, n, cap, 5, P.make_targets([slot.endpoint(env, 0)]))
        assert comp.last_stats()["status"] == 0
        slots.append(slot)
        touched |= x != 0
        scale = torch.tensor(0.3, dtype=torch.float32, device="cuda")
        want = torch.where(x != 0, (want.float() + (-scale if what == "sgd_shadow" else scale) * x).to(dt), want)
    src = P.make_sources([s.endpoint(env, 0) for s in slots], [5] * nsrc)
    args = (P.args_update(_lib.OP_SGD, out, 0.3, shadow=shadow) if what == "sgd_shadow" else P.args_add(out, 0.3))
    P.apply_sparse(env, src, n, args, st)
    env.flush()
    assert st.value == 0 and torch.equal(out, want)
    if shadow is not None:
        assert torch.equal(shadow, torch.where(touched, want.to(torch.bfloat16), torch.zeros_like(shadow)))
    env.close()


@pytest.mark.parametrize("op", ["sgd", "sgd_wd", "momentum", "adamw"])
@pytest.mark.parametrize("shadow", [False, True])
def test_apply_fused_updates(world, op, shadow):
    e0 = world.envs[0]
    dev, n = world.device, 30011
    src, dense = _fill_slots(world, n, 4, seed=5)
    g = torch.zeros(n)
    for d in dense:
        g += d
    g *= 0.25
    w0, m0, v0 = torch.randn(n), 0.1 * torch.randn(n), 0.01 * torch.rand(n) + 0.01
    w, m, v = w0.clone().to(dev), m0.clone().to(dev), v0.clone().to(dev)
    sh = w0.to(torch.bfloat16).to(dev) if shadow else None  # the shadow starts in sync, as in real use
    st = e0.new_status("t")
    lr, mu, wd, b1, b2, eps, step = 0.1, 0.9, 0.01, 0.9, 0.999, 1e-8, 3
    if op == "sgd":
        args = P.args_update(_lib.OP_SGD, w, 0.25, shadow=sh)
        want_w = w0 - g
    elif op == "sgd_wd":
        args = P.args_update(_lib.OP_SGD, w, 0.25, shadow=sh, wd=wd)
        want_w = (1 - wd) * w0 - g
    elif op == "momentum":
        args = P.args_update(_lib.OP_MOMENTUM, w, 0.25, shadow=sh, m=m, lr=lr, momentum=mu, wd=wd)
        want_m = mu * m0 + lr * g
        want_w = (1 - wd) * w0 - want_m
    else:
        args = P.args_update(_lib.OP_ADAMW, w, 0.25, shadow=sh, m=m, v=v, lr=lr, beta1=b1, beta2=b2, eps=eps,
                             wd=wd, step=step)
        want_m = b1 * m0 + (1 - b1) * g
        want_v = b2 * v0 + (1 - b2) * g * g
        want_w = w0 * (1 - lr * wd) - lr * (want_m / (1 - b1 ** step)) / ((want_v / (1 - b2 ** step)).sqrt() + eps)
    P.apply_sparse(e0, src, n, args, st)
    e0.flush()
    assert st.value == 0
    torch.testing.assert_close(w.cpu(), want_w, rtol=1e-5, atol=1e-6)
    if op in ("momentum", "adamw"):
        torch.testing.assert_close(m.cpu(), want_m, rtol=1e-5, atol=1e-7)
    if op == "adamw":
        torch.testing.assert_close(v.cpu(), want_v, rtol=1e-5, atol=1e-8)
    if shadow:
        assert torch.equal(sh.cpu(), w.cpu().to(torch.bfloat16))


@pytest.mark.gpu
@pytest.mark.parametrize("stages", ["1", "2"])
@pytest.mark.parametrize("op", ["sgd_wd", "momentum", "adamw"])
@pytest.mark.parametrize("n", [1024, 30011, (1 << 20) + 77])
def test_apply_bulk_copy_kernel_matches_register_kernel(monkeypatch, n, op, stages):
    """The opt-in dense update that stages w / m / v through shared memory with bulk copies
    (cp.async.bulk + mbarrier) gives the bits of the default kernel."""
    results = []
    for bulk in ("0", "1"):
        monkeypatch.setenv("COMPREX_APPLY_BULK", bulk)
        monkeypatch.setenv("COMPREX_APPLY_STAGES", stages)
        world = cx.LoopbackWorld(2, device="cuda", timeout_ms=2000)
        e0 = world.envs[0]
        src, _ = _fill_slots(world, n, 5, seed=9)
        g = torch.Generator().manual_seed(n)
        w = torch.randn(n, generator=g).cuda()
        m = (0.1 * torch.randn(n, generator=g)).cuda()
        v = (0.01 * torch.rand(n, generator=g) + 0.01).cuda()
        sh = w.to(torch.bfloat16)
        st = e0.new_status("t")
        code = {"sgd_wd": _lib.OP_SGD, "momentum": _lib.OP_MOMENTUM, "adamw": _lib.OP_ADAMW}[op]
        args = P.args_update(code, w, 0.2, shadow=sh, m=None if op == "sgd_wd" else m, v=v if op == "adamw" else None,
                             lr=0.05, momentum=0.9, wd=0.01, step=4)
        for _ in range(2):
            P.apply_sparse(e0, src, n, args, st)
        e0.flush()
        assert st.value == 0
        results.append((w.cpu(), m.cpu(), v.cpu(), sh.cpu()))
        world.close()
    for a, b in zip(*results):
        assert torch.equal(a, b)


@pytest.mark.parametrize("graph", [False, True])
def test_recorded_sequence_with_lanes_and_graph(world, graph):
    """Six independent threshold + compress pairs on side-stream lanes, joined by one apply:
    recorded once, replayed three times (as an op list, and on a GPU as a CUDA graph whose
    kernels take the sequence number from a device cell); equals the direct launches."""
    from comprex_b200.allreduce import _OpSeq
    e0, e1 = world.envs
    dev, nchunk, k = world.device, 3000, 6
    torch.manual_seed(11)
    g = torch.randn(k * nchunk).to(dev)
    slots = [[P.SparseSlot.create(e, nchunk, nchunk) for e in world.envs] for _ in range(k)]
    comps = [P.Compressor(e0, nchunk) for _ in range(k)]
    outs = [torch.zeros(nchunk, device=dev) for _ in range(k)]
    rests = [torch.zeros(k * nchunk, device=dev) for _ in range(2)]
    st = e1.new_status("t")

    def launches(r, seq):
        for c in range(k):
            view, rv = g[c * nchunk:(c + 1) * nchunk], r[c * nchunk:(c + 1) * nchunk]
            with P.lane(e0, c + 1):
                comps[c].threshold_topk(view, rv, nchunk, 0.05)
                comps[c].compress(view, rv, nchunk, nchunk, seq, P.make_targets([slots[c][1].endpoint(e0, 1)]))
        for c in range(k):
            with P.lane(e0, c + 1):
                P.apply_sparse(e0, P.make_sources([slots[c][1].endpoint(e0, 1)], [seq]), nchunk,
                               P.args_add(outs[c]), st)

    e0._rec = rec = []
    try:
        launches(rests[0], 0)
    finally:
        e0._rec = None
    assert len(rec) == 3 * k and {op.lane for op in rec} == set(range(1, k + 1))
    seq_obj = _OpSeq(e0, rec, graph=graph)
    assert (seq_obj.graph is not None) == (graph and e0.dev == _lib.DEV_CUDA)
    for step in (1, 2, 3):
        seq_obj.run(step)
    e0.flush()
    got = torch.cat(outs).cpu()
    for o in outs:
        o.zero_()
    for step in (4, 5, 6):                      # the same launches issued directly
        launches(rests[1], step)
    e0.flush()
    assert st.value == 0
    assert torch.equal(torch.cat(outs).cpu(), got)
    assert torch.equal(rests[0].cpu(), rests[1].cpu())
    assert float(got.abs().sum()) > 0


def test_apply_timeout_sets_status_and_leaves_output(world):
    """A notification that never arrives: the wait gives up, the output is untouched."""
    e0 = world.envs[0]
    n = 2048
    slot = [P.SparseSlot.create(e, n, n) for e in world.envs][0]
    out = torch.ones(n, device=world.device)
    st = e0.new_status("waiter")
    P.apply_sparse(e0, P.make_sources([slot.endpoint(e0)], [1]), n, P.args_add(out), st)
    with pytest.raises(cx.ComprexError, match="TIMEOUT"):
        e0.flush()
    assert torch.equal(out.cpu(), torch.ones(n))
    e0.flush()  # the status word was cleared, the context is still usable
    comp = P.Compressor(e0, n)
    comp.set_threshold(0.0)
    comp.compress(out, None, n, n, 1, P.make_targets([slot.endpoint(e0)]))
    P.apply_sparse(e0, P.make_sources([slot.endpoint(e0)], [1]), n, P.args_add(out), st)
    e0.flush()
    assert torch.equal(out.cpu(), 2 * torch.ones(n))


def test_pushing_reduce_timeout_leaves_counters_clean(world):
    """A pushing reduce whose source never arrives reports TIMEOUT, publishes nothing and leaves
    the completion counters at zero, so that the same launch works when the sender is there."""
    e0, e1 = world.envs
    n = 5000
    src_slot = [P.DenseSlot.create(e, 4 * n) for e in world.envs][0]
    dst_slot = [P.DenseSlot.create(e, 4 * n) for e in world.envs][0]
    own = torch.ones(n, device=world.device)
    out = torch.zeros(n, device=world.device)
    st = e0.new_status("reducer")
    counters = e0.scratch(int(e0.lib.cx_sizeof(4)))
    push = P.make_targets([dst_slot.endpoint(e0, 1)])

    def reduce(seq):
        P.dense_reduce(e0, out, own, n, P.make_sources([src_slot.endpoint(e0)], [seq]), st, push=push,
                       push_seq=seq, counters=counters)
    reduce(1)
    with pytest.raises(cx.ComprexError, match="TIMEOUT"):
        e0.flush()
    assert int(counters.view(torch.int32)[:64].abs().sum()) == 0          # done and the failure mark
    assert e1.read_header(dst_slot.endpoint(e1).hdr).seq == 0             # nothing was published
    sender_counters = e1.scratch(int(e1.lib.cx_sizeof(4)))
    P.dense_send(e1, 2 * torch.ones(n, device=world.device), None, n, 1,
                 P.make_targets([src_slot.endpoint(e1, 0)]), sender_counters)
    e1.flush()
    reduce(1)
    e0.flush()
    assert torch.equal(out.cpu(), 3 * torch.ones(n))
    assert e1.read_header(dst_slot.endpoint(e1).hdr).seq == 1
    assert int(counters.view(torch.int32)[:64].abs().sum()) == 0


def test_apply_rejects_corrupt_header_and_index(world):
    """Host-written garbage in a local slot is reported, never dereferenced."""
    e0 = world.envs[0]
    n = 3000
    slot = [P.SparseSlot.create(e, n, n) for e in world.envs][0]
    x = torch.zeros(n, device=world.device)
    x[5] = 1.0
    comp = P.Compressor(e0, n)
    comp.set_threshold(0.0)
    comp.compress(x, None, n, n, 1, P.make_targets([slot.endpoint(e0)]))
    e0.flush()
    ep = slot.endpoint(e0)
    bad_pair = (C.c_int32 * 2)(2_000_000, 0x3F800000)
    if world.device.type == "cuda":
        _lib.check(e0.lib.cx_cuda_memcpy(ep.pairs, bad_pair, 8, 1, None))
        torch.cuda.synchronize()
    else:
        C.memmove(ep.pairs, bad_pair, 8)
    out = torch.zeros(n, device=world.device)
    st = e0.new_status("decoder")
    P.apply_sparse(e0, P.make_sources([ep], [1]), n, P.args_add(out), st)
    with pytest.raises(cx.ComprexError, match="BAD_INDEX"):
        e0.flush()
    assert float(out.abs().sum()) == 0.0
    # wrong length in the header
    P.apply_sparse(e0, P.make_sources([ep], [1]), n + 1, P.args_add(torch.zeros(n + 1, device=world.device)), st)
    with pytest.raises(cx.ComprexError, match="BAD_HEADER"):
        e0.flush()


@pytest.mark.parametrize("n", [1, 5, 1000, 4099, 65537])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_dense_send_reduce(world, n, dtype):
    e0, e1 = world.envs
    dev = world.device
    es = torch.empty(0, dtype=dtype).element_size()
    slots = [[P.DenseSlot.create(e, n * es) for e in world.envs] for _ in range(2)]
    ctr = e0.scratch(64)
    a, b = torch.randn(n).to(dtype), torch.randn(n).to(dtype)
    own = torch.randn(n).to(dtype)
    P.dense_send(e0, a.to(dev), None, n, 1, P.make_targets([slots[0][1].endpoint(e0, 1)]), ctr)
    P.dense_send(e0, b.to(dev), None, n, 1, P.make_targets([slots[1][1].endpoint(e0, 1)]), ctr)
    st = e1.new_status("t")
    out = own.clone().to(dev)
    src = P.make_sources([slots[0][1].endpoint(e1), slots[1][1].endpoint(e1)], [1, 1])
    P.dense_reduce(e1, out, out, n, src, st, scale=0.5)
    want = ((own.float() + a.float() + b.float()) * 0.5).to(dtype)
    assert torch.equal(out.cpu(), want)
    cp = torch.empty(n, dtype=dtype, device=dev)
    P.dense_reduce(e1, cp, None, n, P.make_sources([slots[0][1].endpoint(e1)], [1]), st)
    assert torch.equal(cp.cpu(), a)
    e1.flush()


def test_dense_send_with_residual_is_compressor_none(world):
    e0, e1 = world.envs
    dev, n = world.device, 3001
    slot = [P.DenseSlot.create(e, 4 * n) for e in world.envs][1]
    g, r0 = torch.randn(n), torch.randn(n)
    r = r0.clone().to(dev)
    P.dense_send(e0, g.to(dev), r, n, 1, P.make_targets([slot.endpoint(e0, 1)]), e0.scratch(64))
    out = torch.empty(n, device=dev)
    P.dense_reduce(e1, out, None, n, P.make_sources([slot.endpoint(e1)], [1]), e1.new_status("t"))
    assert torch.equal(out.cpu(), g + r0)
    assert float(r.abs().sum()) == 0.0


def test_rle_roundtrip_and_residual():
    """Corrected RLE codec: round trip with a threshold above zero, plus error feedback."""
    torch.manual_seed(1)
    n = 1000
    g, r0 = torch.randn(n), 0.2 * torch.randn(n)
    r = r0.clone()
    payload = cx.CompressorRLE.encode(g, r, 1.0)
    v = g + r0
    keep = v.abs() >= 1.0
    out = torch.full((n,), 9.0)
    cx.CompressorRLE.decode(payload, out)
    assert torch.equal(out, torch.where(keep, v, torch.zeros(n)))
    assert torch.equal(r, torch.where(keep, torch.zeros(n), v))
    acc = torch.ones(n)
    cx.CompressorRLE.decode(payload, acc, add=True)
    assert torch.equal(acc, 1 + torch.where(keep, v, torch.zeros(n)))
    # the sparse test vector of test/compressor.cpp (75 % zeros, threshold 0)
    x = torch.arange(16).float() * (torch.arange(16) % 4 == 0)
    out = torch.empty(16)
    cx.CompressorRLE.decode(cx.CompressorRLE.encode(x, None, 0.0), out)
    assert torch.equal(out, x)


@pytest.mark.parametrize("n", [1, 7, 2047, 2048, 2049, 4096, 10007, 70001])
@pytest.mark.parametrize("thr,density", [(0.0, 0.25), (0.8, 1.0), (3.5, 1.0), (100.0, 1.0)])
def test_rle_fused_codec_matches_host_bytes(world, n, thr, density):
    """Fused RLE send/receive (kernels on a GPU, host twin on the CPU): the bytes that land in
    the receiver's slot equal the host codec's payload, the expansion equals the plain
    restatement, the residual keeps what was not sent, and `add` accumulates."""
    e0, e1 = world.envs
    codecs = [P.RleCodec(e, n) for e in world.envs]
    torch.manual_seed(n)
    g = torch.randn(n) * (torch.rand(n) < density)
    r0 = 0.3 * torch.randn(n) * (torch.rand(n) < density)
    cell = torch.full((1,), thr, dtype=torch.float32, device=e0.device)
    gd, r = g.to(e0.device), r0.clone().to(e0.device)
    codecs[0].send(gd, r, cell, 1, 1)
    status = e1.new_status("t")
    out = torch.full((n,), 9.0, device=e1.device)
    codecs[1].recv(out, 1, False, status)
    e1.flush()
    assert status.value == 0
    v = g + r0
    keep = (v.abs() >= thr) & ~((thr == 0.0) & (v == 0))
    assert torch.equal(out.cpu(), torch.where(keep, v, torch.zeros(n)))
    assert torch.equal(r.cpu(), torch.where(keep, torch.zeros(n), v))
    rh = r0.clone()
    expect = cx.CompressorRLE.encode(g, rh, thr)
    ep = codecs[1].slots[1].endpoint(e1)
    hdr = e1.read_header(ep.hdr)
    assert (hdr.kind, hdr.n, hdr.bytes, hdr.nnz) == (_lib.KIND_RLE, n, len(expect), int(keep.sum()))
    assert e1.read_bytes(ep.pairs, len(expect)) == expect
    # second payload (other parity) accumulated on top
    codecs[0].send(None, r, cell.zero_(), 2, 1)            # flush of the residual at threshold 0
    acc = torch.ones(n, device=e1.device)
    codecs[1].recv(acc, 2, True, status)
    e1.flush()
    assert status.value == 0
    assert torch.equal(acc.cpu(), 1 + torch.where(keep, torch.zeros(n), v))
    assert float(r.abs().sum()) == 0.0


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1 << 20, (1 << 20) + 1, 592 * 2048, 592 * 2048 + 1, 3 * 592 * 2048 - 5])
@pytest.mark.parametrize("kind", ["dense", "sparse", "one_run", "alternating"])
def test_rle_chunks_and_run_blocks(n, kind):
    """Several tiles per sending CTA and many blocks of runs per receiving CTA, up to runs longer
    than a CTA's share of the output and the worst case of n runs: the bytes in the slot are the
    host codec's, the expansion (both modes) is exact."""
    world = cx.LoopbackWorld(2, device="cuda", timeout_ms=2000)
    e0, e1 = world.envs
    codecs = [P.RleCodec(e, n) for e in world.envs]
    gen = torch.Generator().manual_seed(n)
    g = torch.randn(n, generator=gen)
    thr = {"dense": 1.0, "sparse": 3.5, "one_run": 100.0, "alternating": 0.5}[kind]
    if kind == "alternating":
        g = torch.where(torch.arange(n) % 2 == 0, g.abs() + 1.0, torch.zeros(n))
    cell = torch.full((1,), thr, dtype=torch.float32, device="cuda")
    r = torch.zeros(n, device="cuda")
    codecs[0].send(g.cuda(), r, cell, 1, 1)
    status = e1.new_status("t")
    out = torch.full((n,), 9.0, device="cuda")
    codecs[1].recv(out, 1, False, status)
    acc = torch.ones(n, device="cuda")
    codecs[1].recv(acc, 1, True, status)
    e1.flush()
    assert status.value == 0
    kept = torch.where(g.abs() >= thr, g, torch.zeros(n))
    assert torch.equal(out.cpu(), kept) and torch.equal(acc.cpu(), 1 + kept)
    assert torch.equal(r.cpu(), g - kept)
    expect = cx.CompressorRLE.encode(g, torch.zeros(n), thr)
    ep = codecs[1].slots[1].endpoint(e1)
    assert e1.read_header(ep.hdr).bytes == len(expect) and e1.read_bytes(ep.pairs, len(expect)) == expect
    world.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 32, 33, 1023, 1024, 1025, 8 * 1024 - 1, 8 * 1024 + 1, 4736 * 1024 + 1])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", ["edges", "runs", "none"])
def test_rle_run_starts_at_chunk_edges(n, dtype, shape):
    """Runs that begin, end or go on where a row, a sub-tile, a warp's chunk or a CTA's chunks meet (the
    element in front decides), views at odd addresses, with and without a residual: payload bytes of the
    host codec."""
    world = cx.LoopbackWorld(2, device="cuda", timeout_ms=2000)
    e0, e1 = world.envs
    codecs = [P.RleCodec(e, n) for e in world.envs]
    at = torch.arange(n)
    keep = {"edges": (at % 32 == 31) | (at % 1024 == 0) | (at % 8192 == 8191), "runs": (at // 1024) % 2 == 1,
            "none": torch.zeros(n, dtype=torch.bool)}[shape]
    g = torch.where(keep, torch.full((n,), 2.0), torch.full((n,), 0.25)).to(dtype)
    cell = torch.full((1,), 1.0, dtype=torch.float32, device="cuda")
    status = e1.new_status("t")
    for seq, with_r in ((1, True), (2, False)):
        gd = torch.zeros(n + 1, dtype=dtype, device="cuda")[1:].copy_(g)
        r = torch.zeros(n + 1, device="cuda")[1:].fill_(0.125) if with_r else None
        codecs[0].send(gd, r, cell, seq, 1)
        out = torch.full((n + 1,), 9.0, device="cuda")[1:]
        codecs[1].recv(out, seq, False, status)
        e1.flush()
        assert status.value == 0
        rh = torch.full((n,), 0.125) if with_r else None
        expect = cx.CompressorRLE.encode(g.float(), rh, 1.0)
        ep = codecs[1].slots[seq & 1].endpoint(e1)
        assert e1.read_header(ep.hdr).bytes == len(expect) and e1.read_bytes(ep.pairs, len(expect)) == expect
        v = g.float() + (0.125 if with_r else 0.0)
        assert torch.equal(out.cpu(), torch.where(keep, v, torch.zeros(n)))
        if with_r:
            assert torch.equal(r.cpu(), rh)
    world.close()


def test_rle_fused_receive_rejects_corrupt_runs(world):
    """Host-side fault injection: run lengths that do not add up to n set BAD_HEADER and leave
    the output untouched; a payload that never arrives times out with a status."""
    e0, e1 = world.envs
    n = 5000
    codecs = [P.RleCodec(e, n) for e in world.envs]
    g = torch.randn(n, generator=torch.Generator().manual_seed(0))
    cell = torch.full((1,), 1.0, dtype=torch.float32, device=e0.device)
    codecs[0].send(g.to(e0.device), None, cell, 1, 1)
    e0.flush()
    ep = codecs[1].slots[1].endpoint(e1)
    hdr = e1.read_header(ep.hdr)
    raw = bytearray(e1.read_bytes(ep.pairs, hdr.bytes))
    runs_at = 16 + 4 * hdr.nnz
    first = int.from_bytes(raw[runs_at:runs_at + 4], "little")
    raw[runs_at:runs_at + 4] = (first + 1).to_bytes(4, "little")       # one element too many
    t = torch.frombuffer(raw, dtype=torch.uint8)
    if e1.dev == _lib.DEV_CUDA:
        _lib.check(e1.lib.cx_cuda_memcpy(ep.pairs, t.data_ptr(), len(raw), 1, None), "memcpy")
    else:
        C.memmove(ep.pairs, t.data_ptr(), len(raw))
    status = e1.new_status("t")
    out = torch.full((n,), 9.0, device=e1.device)
    codecs[1].recv(out, 1, False, status)
    with pytest.raises(cx.ComprexError, match="BAD_HEADER"):
        e1.flush()
    assert torch.equal(out.cpu(), torch.full((n,), 9.0))
    status2 = e1.new_status("t2")
    codecs[1].recv(out, 2, False, status2)                 # nobody sent payload 2
    with pytest.raises(cx.ComprexError, match="TIMEOUT"):
        e1.flush()
    assert torch.equal(out.cpu(), torch.full((n,), 9.0))


@pytest.mark.gpu
@pytest.mark.parametrize("samples", [1, 2, 31, 33, 255, 256, 257, 1000, 1024, 1025, 2047, 2048, 2049])
@pytest.mark.parametrize("ratio", [0.001, 0.01, 0.03, 0.1, 0.999])
@pytest.mark.parametrize("kind", ["gauss", "ties", "equal", "zeros"])
def test_threshold_of_small_samples(samples, ratio, kind):
    """The sampled threshold for samples on both sides of the kernel's rounds and of its limit, ranks on both
    sides of its two selections, and keys with so many ties that the candidates do not fit: the reference's
    value, from a vector of exactly that many elements and from a longer one."""
    env = cx.GaspiEnvironment(1 << 16, device="cuda")
    for n in (samples, 7 * samples + 3):
        gen = torch.Generator().manual_seed(samples)
        x = torch.randn(n, generator=gen)
        if kind == "ties":
            x = torch.randint(-3, 4, (n,), generator=gen).float()
        elif kind == "equal":
            x = torch.full((n,), -1.5)
        elif kind == "zeros":
            x = torch.where(torch.rand(n, generator=gen) < 0.99, torch.zeros(n), x)
        comp = P.Compressor(env, n)
        comp.threshold_topk(x.cuda(), None, n, ratio, samples, 0.0)
        env.flush()
        assert float(comp.thr) == ref_threshold_topk(x, ratio, samples, 0.0)
    env.close()


@pytest.mark.gpu
@pytest.mark.parametrize("count", [0, 1, 33, 511, 512, 513, 1023, 1024])
@pytest.mark.parametrize("room", [1, 32, 511, 512, 513, 700, 1024])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_dense_subtiles_and_full_slots(count, room, dtype):
    """One sub-tile with `count` survivors into a slot with room for `room`: around the length of the warp's
    list, and cut off inside each of its parts.  What is stored and what stays add up to the vector, with
    and without a gradient, and nothing else is touched."""
    n = 1024
    world = cx.LoopbackWorld(1, device="cuda", timeout_ms=2000)
    e0 = world.envs[0]
    cap, gen = room, torch.Generator().manual_seed(count)
    big = torch.zeros(n, dtype=torch.bool)
    big[torch.randperm(n, generator=gen)[:count]] = True
    g = torch.where(big, 2.0 + torch.rand(n, generator=gen), 0.25 * torch.rand(n, generator=gen)).to(dtype)
    comp = P.Compressor(e0, n)
    for seq, with_g in ((1, True), (2, False)):
        slot = P.SparseSlot.create(e0, n, cap)
        r0 = 0.125 * torch.ones(n) if with_g else g.float()
        v = g.float() + r0 if with_g else r0
        r = r0.cuda()
        comp.set_threshold(1.0)
        comp.compress(g.cuda() if with_g else None, r, n, cap, seq, P.make_targets([slot.endpoint(e0)]))
        e0.flush()
        hdr, idx, val = read_pairs(e0, slot)[:3]
        assert (hdr.nnz, hdr.nnz_found) == (min(count, cap), count)
        sent = torch.zeros(n)
        sent[idx.long()] = val
        assert idx.unique().numel() == min(count, cap) and bool(big[idx.long()].all())
        assert torch.equal(sent + r.cpu(), v) and bool((sent * r.cpu() == 0).all())
    world.close()


@pytest.mark.gpu
@pytest.mark.parametrize("extra", [0, 1024, 1024 + 500])
@pytest.mark.parametrize("counts", [(0, 47, 48, 49), (1024, 500, 10, 0), (511, 512, 513, 48)])
@pytest.mark.parametrize("room", [1.0, 0.7])
def test_dense_subtiles_of_long_vectors(extra, counts, room):
    """fp32 vectors on both sides of the length from which sub-tiles with many survivors are listed another way: all
    of them, none, numbers around the line and around the length of the warp's list, and slots that are too small."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    subs = 16 * 16 * sms                       # 16 sub-tiles for each of 16 warps per SM
    n = 1024 * subs + extra
    env = cx.GaspiEnvironment(1 << 16, device="cuda")
    e0 = env.get()
    gen = torch.Generator(device="cuda").manual_seed(extra)
    score = torch.rand(subs, 1024, device="cuda", generator=gen)
    want = torch.tensor(counts, device="cuda").repeat(subs)[:subs]
    kth = score.sort(dim=1).values
    big = score <= torch.where(want > 0, kth.gather(1, (want - 1).clamp(min=0)[:, None])[:, 0], -1.0)[:, None]
    big = torch.cat((big.view(-1), torch.ones(extra, dtype=torch.bool, device="cuda")))
    del score, kth
    g = torch.where(big, 2.0, 0.25) + 0.125 * torch.rand(n, device="cuda", generator=gen)
    r = torch.rand(n, device="cuda", generator=gen) * 0.125
    v = r + g
    cap = n + 32 * 1024 if room == 1.0 else int(room * int(big.sum()))      # (the regions of a slot fill unevenly)
    comp, slot = P.Compressor(e0, n), P.SparseSlot.create(e0, n, cap)
    comp.set_threshold(1.0)
    comp.compress(g, r, n, cap, 1, P.make_targets([slot.endpoint(e0)]))
    out, status = torch.full((n,), 9.0, device="cuda"), e0.new_status("t")
    P.apply_sparse(e0, P.make_sources([slot.endpoint(e0)], [1]), n, P.args_set(out), status)
    e0.flush()
    hdr = e0.read_header(slot.endpoint(e0).hdr)
    sent = out != 0
    assert status.value == 0 and hdr.nnz_found == int(big.sum()) and hdr.nnz == int(sent.sum())
    assert bool((sent <= big).all()) and torch.equal(out + r, v) and not bool(r[sent].any())
    if room == 1.0:
        assert torch.equal(sent, big)
    env.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 1000, 1023, 8 * 1024, 8 * 1024 + 1, 100003, 296 * 8 * 1024, 296 * 8 * 1024 + 1])
@pytest.mark.parametrize("ratio", [0.001, 0.01, 0.1, 0.7])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_threshold_and_compress_as_one_list(n, ratio, dtype):
    """The op list [threshold, compress] (the compress kernel loads ahead of the threshold) gives
    threshold, payload and residual of the two launches issued one by one, call after call; views at
    odd addresses too."""
    world = cx.LoopbackWorld(2, device="cuda", timeout_ms=2000)
    e0, e1 = world.envs
    gen = torch.Generator(device="cuda").manual_seed(n)
    slots = [[P.SparseSlot.create(e, n, n) for e in world.envs][1] for _ in range(2)]
    comps = [P.Compressor(e0, n) for _ in range(2)]
    for shift in (0, 1):
        rs = [torch.randn(n + 1, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))[shift:shift + n].mul(0.5)
              for _ in range(2)]
        if shift:
            rs = [torch.cat((torch.zeros(1, device="cuda"), r))[1:] for r in rs]
        for seq in (1, 2, 3):
            g = torch.randn(n + 1, device="cuda", generator=gen).to(dtype)[shift:shift + n]
            comps[0].threshold_topk(g, rs[0], n, ratio)
            comps[0].compress(g, rs[0], n, n, seq, P.make_targets([slots[0].endpoint(e0, 1)]))
            ops = (_lib.Op * 2)(*comps[1].send_ops(rs[1], n, n, P.make_targets([slots[1].endpoint(e0, 1)]), ratio, 1000, 10.0))
            for o in ops:
                o.g, o.dtype = g.data_ptr(), _lib.dtype_code(dtype)
            _lib.check(e0.lib.cx_run_ops(ops, 2, seq, _lib.stream_ptr(e0.device)))
            e0.flush()
            assert torch.equal(comps[0].thr, comps[1].thr)
            a, b = (read_pairs(e1, s) for s in slots)
            assert a[0].seq == b[0].seq == seq and a[0].nnz == b[0].nnz and a[0].nnz_found == b[0].nnz_found
            for x, y in zip(a[1:], b[1:]):
                assert torch.equal(x, y)
            assert torch.equal(rs[0], rs[1])
    world.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1000, 4096, 100003, (1 << 22) + 5])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_cuda_kernels_match_host_bitwise(n, dtype):
    """threshold + compress + apply on the GPU produce the bits of the host implementation
    (the AdamW weights to within the hardware's approximate square root and reciprocal)."""
    torch.manual_seed(n)
    g = torch.randn(n).to(dtype)
    r0 = 0.7 * torch.randn(n)
    w0 = torch.randn(n)
    res = {}
    for dev in ("cpu", "cuda"):
        world = cx.LoopbackWorld(2, device=dev)
        e0, e1 = world.envs
        cap = n // 8
        slot = [P.SparseSlot.create(e, n, cap) for e in world.envs][1]
        comp = P.Compressor(e0, n)
        r = r0.clone().to(dev)
        comp.threshold_topk(g.to(dev), r, n, 0.02)
        comp.compress(g.to(dev), r, n, cap, 1, P.make_targets([slot.endpoint(e0, 1)]))
        hdr, idx, val, prefix = read_pairs(e1, slot)
        w = w0.clone().to(dev)
        m = torch.zeros(n, device=dev)
        v = torch.zeros(n, device=dev)
        sh = torch.zeros(n, dtype=torch.bfloat16, device=dev)
        st = e1.new_status("t")
        P.apply_sparse(e1, P.make_sources([slot.endpoint(e1)], [1]), n,
                       P.args_update(_lib.OP_ADAMW, w, 0.5, shadow=sh, m=m, v=v, lr=0.01, wd=0.1, step=2), st)
        e1.flush()
        res[dev] = (comp.thr.cpu().clone(), idx, val, prefix, r.cpu(), w.cpu(), m.cpu(), v.cpu(), sh.cpu())
        world.close()
    names = ["thr", "idx", "val", "prefix", "r", "w", "m", "v", "shadow"]
    for name, a, b in zip(names, res["cpu"], res["cuda"]):
        if name == "w":        # the kernel's AdamW step uses the approximate sqrt / reciprocal units
            torch.testing.assert_close(b, a, rtol=1e-6, atol=1e-6)
        elif name == "shadow":
            torch.testing.assert_close(b.float(), a.float(), rtol=1e-2, atol=1e-7)
        else:
            assert torch.equal(a, b), name
