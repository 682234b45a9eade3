"""Parity of the DSA top-k indexer's CUDA path (through the C ABI) against its oracle.  Needs a B200."""
import ctypes
import os

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def _run(pkg, inputs):
    q, cache, w, sl, table = (t.to(DEV) for t in inputs)
    out = torch.full((q.shape[0], 2048), -7, dtype=torch.int32, device=DEV)
    pkg.run_dsa_topk_indexer(q, cache, w, sl, table, out)
    pkg.dsa_check()
    return out


@pytest.mark.parametrize("name", ["dsa_small", "dsa_cut", "dsa_long"])
def test_indexer_matches_reference_entry_point_vectors(name, pkg, golden_dir):
    """Against the stored outputs of the reference's own entry point: the same tokens, best first; tokens whose
    scores differ by less than 2e-5 of the largest score may swap places (the tensor core sums the 128 products of a
    head in another order than the host's matrix product, the sum over the heads likewise)."""
    from oracle import dsa_oracle
    g = torch.load(os.path.join(golden_dir, name + ".pt"))
    inputs = dsa_oracle.make_inputs(**g["make_inputs"])
    _, scores = dsa_oracle.topk_indexer(*inputs)
    out = _run(pkg, inputs)
    ok, stats = dsa_oracle.check_topk(out, g["topk_indices"], scores, inputs[3], inputs[4])
    assert ok, stats
    # sequences no longer than 2048 keep every token: exactly the same set as the reference
    for b, n in enumerate(g["make_inputs"]["seq_lens"]):
        if 0 < n <= 2048:
            assert set(out[b, :n].tolist()) == set(g["topk_indices"][b, :n].tolist())
        if n == 0:
            assert bool((out[b] == -1).all())


@pytest.mark.parametrize("seq_lens,seed", [([40000, 3, 17000, 2048, 70000], 11), ([128] * 40, 12)])
def test_indexer_matches_oracle(seq_lens, seed, pkg):
    """Long sequences (several radix passes with many candidates per byte) and a wide batch, against the oracle
    evaluated with torch on the GPU."""
    from oracle import dsa_oracle
    inputs = tuple(t.to(DEV) for t in dsa_oracle.make_inputs(seq_lens, seed=seed))
    want, scores = dsa_oracle.topk_indexer(*inputs)
    out = _run(pkg, inputs)
    ok, stats = dsa_oracle.check_topk(out, want, scores, inputs[3].cpu(), inputs[4].cpu())
    assert ok, stats
    assert stats["most_tokens_swapped_at_the_cut"] <= 4


def test_indexer_ties_and_determinism(pkg):
    """All keys equal: every score is the same, so the cut is one big tie; the lowest positions win, in position
    order, run after run."""
    from oracle import dsa_oracle
    q, cache, w, sl, table = dsa_oracle.make_inputs([5000], seed=13)
    cache = cache.view(torch.uint8).reshape(cache.shape[0], -1).clone()
    cache[:] = cache[0, :132].repeat(64)[: cache.shape[1]] * 0 + cache[0:1]      # every page a copy of page 0
    row0 = cache[:, :128].clone()
    cache[:, : 64 * 128] = row0.repeat(1, 64)                                   # every token a copy of token 0
    cache[:, 64 * 128:] = cache[:, 64 * 128: 64 * 128 + 4].repeat(1, 64)        # ... with token 0's scale
    cache = cache.view(torch.int8).view(-1, 64, 1, 132)
    a = _run(pkg, (q, cache, w, sl, table))
    b = _run(pkg, (q, cache, w, sl, table))
    assert torch.equal(a, b)
    want = (table[0, torch.arange(2048) // 64].to(torch.int64) * 64 + torch.arange(2048) % 64).to(torch.int32)
    assert torch.equal(a[0].cpu(), want)


@pytest.mark.parametrize("lens,table_pages,kind", [
    ([8192, 2049, 2048, 1, 0], 128, "spread"),           # one CTA per sequence: its largest table
    ([8193, 1024, 5000], 129, "spread"),                 # two CTAs
    ([16385, 30000, 7], 512, "spread"),                  # four
    ([65536, 2049], 1024, "spread"),                     # eight, eight positions per thread
    ([65537, 131072], 2048, "spread"),                   # sixteen positions per thread
    ([131073, 300], 2049, "spread"),                     # scores read again in every sweep
    ([3000, 20000, 6000], 512, "zeros"),                 # the cut lies among equal scores: radix select and sort
    ([140000, 9000], 2200, "zeros"),
    ([9000, 4000], 256, "outlier"),                      # one score stretches the range
    ([6000], 94, "nan"),
    # no use for the bins: every CTA of the cluster selects among its own positions, the first one among those
    ([8193, 20000, 9216], 512, "outlier"),               # two and four CTAs, some with 1024 positions
    ([65536, 40000, 8000], 1024, "outlier"),             # eight
    ([131072, 17000], 2048, "outlier"),                  # sixteen positions per thread
    ([131073, 300000], 4700, "outlier"),                 # read again in every pass
    ([65536, 30000], 1024, "zeros"),
    ([30000, 5000], 512, "inf"),                         # the range is not finite
    ([30000, 5000], 512, "nan_weight"),                  # every score of the first sequence is NaN
    ([12000 + 9 * i for i in range(80)], 200, "spread"), # one CTA per sequence, sixteen positions per thread
    ([12000 + 9 * i for i in range(80)], 200, "outlier"),
])
def test_indexer_selection_is_exact(lens, table_pages, kind, pkg):
    """Every branch of the selection, with scores that both sides compute without a rounding difference: one head of
    small integers carries weight 1, so a score is one exact integer times the token's scale.  The reference is a
    stable descending sort (ties by position); indices must be equal."""
    g = torch.Generator(device=DEV).manual_seed(len(lens) + table_pages)
    B, need = len(lens), [(n + 63) // 64 for n in lens]
    pages = sum(need) + 2
    q = torch.randint(-4, 5, (B, 64, 128), generator=g, device=DEV).float()
    keys = torch.randint(-4, 5, (pages, 64, 128), generator=g, device=DEV).float()
    scale = 0.5 + torch.rand(pages, 64, generator=g, device=DEV)
    if kind != "spread":
        scale.fill_(1.0)
    if kind == "zeros":          # three quarters of the keys repeat one key: scores of zero or one large tie
        keys[:, 16:] = -q[0, 0]
    if kind == "outlier":
        scale[0, 0] = 1e7
        keys[0, 0] = q[0, 0]
        scale[need[0], 0] = 1e7                          # and the second sequence's first token
        keys[need[0], 0] = q[1, 0]
    if kind == "inf":
        q[:, 1:] = 0                                     # (a weight of zero times infinity would be NaN)
        scale[0, 0] = float("inf")
        keys[0, 0] = q[0, 0]
    if kind == "nan":
        scale[0, 0] = float("nan")
    cache = torch.empty(pages, 64 * 132, dtype=torch.uint8, device=DEV)
    cache[:, :8192] = keys.to(torch.float8_e4m3fn).view(torch.uint8).view(pages, -1)
    cache[:, 8192:] = scale.view(torch.uint8)
    w = torch.zeros(B, 64, device=DEV)
    w[:, 0] = 1.0
    if kind == "nan_weight":
        w[0, 1] = float("nan")
    perm = torch.arange(pages, device=DEV) if kind in ("outlier", "inf", "nan") else torch.randperm(pages, generator=g, device=DEV)
    table = torch.zeros(B, table_pages, dtype=torch.int32, device=DEV)
    at = 0
    for b, n in enumerate(need):
        table[b, :n] = perm[at: at + n].int()
        at += n
    sl = torch.tensor(lens, dtype=torch.int32, device=DEV)
    out = torch.full((B, 2048), -7, dtype=torch.int32, device=DEV)
    pkg.run_dsa_topk_indexer(q.to(torch.float8_e4m3fn), cache.view(torch.int8).view(pages, 64, 1, 132), w, sl, table, out)
    pkg.dsa_check()
    for b, n in enumerate(lens):
        k = min(n, 2048)
        assert bool((out[b, k:] == -1).all())
        if n == 0:
            continue
        tb = table[b].long()
        score = torch.relu((keys[tb[: need[b]]] @ q[b, 0]) * scale[tb[: need[b]]]).flatten()[:n]
        score = torch.nan_to_num(score, nan=0.0, posinf=float("inf"))      # relu is a maximum with zero in the kernel: a NaN counts as zero
        if kind == "nan_weight" and b == 0:
            score = torch.zeros_like(score)           # all the same: ties by position
        best = torch.sort(score, descending=True, stable=True).indices[:k]
        assert torch.equal(out[b, :k].long(), tb[best // 64] * 64 + best % 64), (b, n)


@pytest.mark.parametrize("lens,table_pages,absent", [
    ([3000, 700, 64], 128, [1, 5, 6]),           # one CTA per sequence; the third has no page at all
    ([30000, 5000], 512, [0, 7, 77, 78, 79]),    # a cluster
    ([140000], 2200, [3, 1000, 2187]),           # scores read again in every sweep
])
def test_indexer_ranks_absent_pages_last(lens, table_pages, absent, pkg):
    """A negative table entry has no keys: its positions are worse than all others and come back as -1.  The call
    before leaves other scores in the scratch buffer, which must not be met again."""
    from oracle import dsa_oracle
    q, cache, w, sl, table = (t.to(DEV) for t in dsa_oracle.make_inputs(lens, seed=5))
    table = torch.nn.functional.pad(table, (0, table_pages - table.shape[1]))
    _run(pkg, (q, cache, w * 1e6, sl, table))
    before = _run(pkg, (q, cache, w, sl, table))
    holes = table.clone()
    for b, n in enumerate(lens):
        pages = [p for p in absent if p < (n + 63) // 64] if b < 2 else list(range((n + 63) // 64))
        holes[b, pages] = torch.tensor([-1 - 70 * p for p in pages], dtype=torch.int32, device=DEV)
    out = _run(pkg, (q, cache, w, sl, holes))
    for b, n in enumerate(lens):
        pos = torch.arange(n, device=DEV)
        left = int((holes[b].long()[pos // 64] >= 0).sum())
        k = min(2048, left)
        assert bool((out[b, k:] == -1).all())
        gone = set((table[b].long()[pos // 64] * 64 + pos % 64)[holes[b].long()[pos // 64] < 0].tolist())
        kept = [t for t in before[b].tolist() if t >= 0 and t not in gone]
        assert out[b, :min(k, len(kept))].tolist() == kept[:k]


@pytest.mark.parametrize("streams", [2, 10])        # ten: more than hold a scratch buffer at a time
def test_indexer_calls_on_several_streams_at_once(streams, pkg):
    """Every stream's call has scores of its own: the outputs are those of the calls one after the other."""
    from oracle import dsa_oracle
    sets = [tuple(t.to(DEV) for t in dsa_oracle.make_inputs([20000 + 64 * i, 900, 9000], seed=20 + i)) for i in range(streams)]
    want = [_run(pkg, s) for s in sets]
    outs = [torch.full_like(w, -7) for w in want]
    side = [torch.cuda.Stream() for _ in range(streams)]
    torch.cuda.synchronize()
    for _ in range(20):
        for s, stream, out in zip(sets, side, outs):
            with torch.cuda.stream(stream):
                pkg.run_dsa_topk_indexer(*s, out)
    torch.cuda.synchronize()
    pkg.dsa_check()
    for w, out in zip(want, outs):
        assert torch.equal(w, out)


def test_indexer_graph_beside_calls_on_other_streams(pkg):
    """A graph captured on a stream that never ran a call keeps its own scores, also while other streams call, and a
    larger call on another stream leaves its buffer alone."""
    from oracle import dsa_oracle
    a, b, c = (tuple(t.to(DEV) for t in dsa_oracle.make_inputs(lens, seed=31 + len(lens))) for lens in ([12000, 70], [9000], [40000, 3, 20000]))
    want = [_run(pkg, x) for x in (a, b, c)]
    outs = [torch.full_like(w, -7) for w in want]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=torch.cuda.Stream()):
        pkg.run_dsa_topk_indexer(*a, outs[0])
    other = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(10):
        graph.replay()
        with torch.cuda.stream(other):
            pkg.run_dsa_topk_indexer(*b, outs[1])
            pkg.run_dsa_topk_indexer(*c, outs[2])
    torch.cuda.synchronize()
    pkg.dsa_check()
    for w, out in zip(want, outs):
        assert torch.equal(w, out)


def _us_per_call(f, calls=20):
    times = []
    for _ in range(5):
        begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        begin.record()
        for _ in range(calls):
            f()
        end.record()
        torch.cuda.synchronize()
        times.append(begin.elapsed_time(end) * 1e3 / calls)
    return min(times[1:])


@pytest.mark.parametrize("length", [65536, 262144])
def test_indexer_cost_without_bins_is_bounded(length, pkg):
    """One outlier takes the bins' use away.  The selection that is left has to stay a matter of the whole cluster: 2.1
    times (65536 tokens) and 2.7 times (262144) the call with separable scores were measured, 6.6 and 13.6 times when one
    CTA read the whole sequence alone."""
    from oracle import dsa_oracle
    q, cache, w, sl, table = (t.to(DEV) for t in dsa_oracle.make_inputs([length], seed=3))
    out = torch.empty(1, 2048, dtype=torch.int32, device=DEV)
    plain = _us_per_call(lambda: pkg.run_dsa_topk_indexer(q, cache, w.abs(), sl, table, out))
    stretched = cache.clone().view(-1, 64 * 132)
    scales = stretched[int(table[0, 5]), 64 * 128:].view(torch.float32)
    scales[7] *= 3e3
    stretched = stretched.view(cache.shape)
    outlier = _us_per_call(lambda: pkg.run_dsa_topk_indexer(q, stretched, w.abs(), sl, table, out))
    assert int(out[0, 0]) == int(table[0, 5]) * 64 + 7
    assert outlier < 4.5 * plain, (outlier, plain)


def test_indexer_argument_validation(pkg):
    from oracle import dsa_oracle
    q, cache, w, sl, table = (t.to(DEV) for t in dsa_oracle.make_inputs([100], seed=1))
    out = torch.empty(1, 2048, dtype=torch.int32, device=DEV)
    with pytest.raises(ValueError, match="topk_indices"):
        pkg.run_dsa_topk_indexer(q, cache, w, sl, table, out[:, :100])
    with pytest.raises(ValueError, match="weights"):
        pkg.run_dsa_topk_indexer(q, cache, w.double(), sl, table, out)
    with pytest.raises(ValueError, match="no CPU path"):
        pkg.run_dsa_topk_indexer(q.cpu(), cache, w, sl, table, out)
    pkg.run_dsa_topk_indexer(q, cache, w, sl, table, out)
    pkg.dsa_check()


@pytest.mark.parametrize("seq_lens", [[3000], [700, 5000, 30000], [65536] * 32])
def test_indexer_calls_that_give_up_halfway_leave_nothing_on_its_way(seq_lens, pkg):
    """Limits around the latency of a load: score CTAs give up with copies and MMAs under way (one, two or eight key tiles
    per CTA) and must see them land before they leave.  The call reports status 201 (a look at a barrier may itself take
    as long as one load, so all but the shortest limit may pass), and the calls behind it give what they gave before."""
    from oracle import dsa_oracle
    inputs = tuple(t.to(DEV) for t in dsa_oracle.make_inputs(seq_lens, seed=14))
    before = _run(pkg, inputs)
    lib = pkg.load_library()
    failed = 0
    for limit in (1, 1, 1, 100, 400, 1000, 3000):
        assert lib.syfi_dsa_debug_wait_limit(ctypes.c_int64(limit)) == 0
        try:
            _run(pkg, inputs)
        except pkg.MoeError as err:
            assert "status 201" in str(err), str(err)
            failed += 1
        assert torch.equal(_run(pkg, inputs), before), limit
    assert failed >= 1, failed
