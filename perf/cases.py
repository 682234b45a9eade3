"""The work this library is used for, as cases that can be timed: the FP8 block-scale MoE layer from one decoded token to
a large prefill (device tensors, pre-packed weights, an expert-parallel rank's f32 partial, host buffers) and the DSA
top-k indexer from a short batch to two million tokens.

A case is a dict of plain values.  ``prepare(case, seed)`` makes what a user's program holds before the call (weights on
the GPU, the step's tensors, the output buffer), ``run(state)`` is one call of the public entry point.
"""
import importlib
import math

import torch

pkg = importlib.import_module("mlsys-contest-syfi-agent-assisted_b200")
workloads = importlib.import_module("mlsys-contest-syfi-agent-assisted_b200.workloads")

DEV = "cuda:0"
HEADS, DIM, PAGE, TOPK = 64, 128, 64, 2048
HOT_EXPERTS, HOT_SEED, HOT_SKEW = 16, 1, 1.5      # the repository's load-imbalance configuration
FEW = 16                                          # batches below this lean towards the local experts, see _logits


# ------------------------------------------------------------------------------------------------- the cases
def _moe(name, tokens, experts=32, offset=0, hot=False, mode="device"):
    """mode: device = run_moe, packed = run_moe_prepacked, partial = run_moe into f32, host = run_moe_host."""
    case = {"op": "moe", "mode": mode, "tokens": tokens, "experts": experts, "offset": offset, "hot": hot}
    return dict(case, name=name) if name else case


def _dsa(name, batch, shortest, longest, table_pages):
    case = {"op": "dsa", "batch": batch, "shortest": shortest, "longest": longest, "table_pages": table_pages}
    return dict(case, name=name) if name else case


def listed():
    return [
        # one sequence being decoded: the smallest call, a chain of launches around one or two experts' weights
        _moe("moe_t1", 1),
        # a decode batch (the benchmark's decode size): streams the active experts' weights
        _moe("moe_t64", 64),
        # a decode batch of no round size in a serving process that packed its weights once at load time
        _moe("moe_t293_packed", 293, mode="packed"),
        # a prefill chunk (the benchmark's chunk size)
        _moe("moe_t1024", 1024),
        # a rank of an expert-parallel job on replicated tokens with hot experts: f32 partial for the sum over ranks
        _moe("moe_t4096_hot_partial", 4096, offset=160, hot=True, mode="partial"),
        # the large prefill of the benchmark, and the largest batch of the repository's sweep
        _moe("moe_t8192", 8192),
        _moe("moe_t16384", 16384),
        # the step's tensors in pinned host memory, as in the benchmark's end-to-end figure: decode and a ragged prefill
        _moe("moe_host_t64", 64, mode="host"),
        _moe("moe_host_t5000", 5000, mode="host"),
        # indexer: a few short sequences, some below the 2048 tokens that are kept, in a table made for longer ones
        _dsa("dsa_b3_short", 3, 700, 5000, 128),
        # indexer: an ordinary decode batch, lengths from hundreds to tens of thousands
        _dsa("dsa_b24_ragged", 24, 300, 30000, 512),
        # indexer: the benchmark's batch, two million tokens
        _dsa("dsa_b32_64k", 32, 65536, 65536, 1024),
    ]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    if rng.random() < 0.3:
        batch = _log_uniform(rng, 1, 40)
        # at most the two million tokens of the largest listed batch
        longest = _log_uniform(rng, 65, min(65536, 2097152 // batch))
        shortest = _log_uniform(rng, max(1, longest // 100), longest)
        used = (longest + PAGE - 1) // PAGE
        return _dsa(None, batch, shortest, longest, rng.choice([used, min(1024, 2 * used), max(used, 128)]))
    mode = rng.choice(["device", "device", "device", "packed", "partial", "host"])
    experts = rng.choice([32, 32, 32, 16, 8])
    offset = 32 * rng.randrange(8)
    hot = mode != "host" and rng.random() < 0.25
    most = {"host": 5000, "packed": 4096}.get(mode, 16384)
    return _moe(None, _log_uniform(rng, 1, min(most, 8192) if hot else most), experts, offset, hot, mode)


# ------------------------------------------------------------------------------------------------- the inputs
def _logits(case, g, device):
    x = torch.randn(case["tokens"], 256, generator=g, device=device)
    if case["hot"]:
        hot = torch.randperm(256, generator=torch.Generator().manual_seed(HOT_SEED))[:HOT_EXPERTS]
        x[:, hot.to(device)] += HOT_SKEW
    if case["tokens"] < FEW:     # a rank is asked with so few tokens because they were routed to experts it holds
        x[:, case["offset"]: case["offset"] + case["experts"]] += 1.0
    bias = (torch.randn(256, generator=g, device=device) * 0.1).to(torch.bfloat16)
    return x, bias


def _prepare_moe(case, seed):
    T, E, H, I = case["tokens"], case["experts"], workloads.HIDDEN, workloads.INTER
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    logits, bias = _logits(case, g, DEV)
    hs, hs_scale = workloads.quantize_act_1x128(
        torch.randn(T, H, generator=g, device=DEV).to(torch.bfloat16))
    f8 = torch.float8_e4m3fn
    w13 = torch.empty(E, 2 * I, H, dtype=f8, device=DEV)
    w13_s = torch.empty(E, 2 * I // 128, H // 128, device=DEV)
    w2 = torch.empty(E, H, I, dtype=f8, device=DEV)
    w2_s = torch.empty(E, H // 128, I // 128, device=DEV)
    for e in range(E):
        w13[e], w13_s[e] = workloads.quantize_weight_128x128(torch.randn(2 * I, H, generator=g, device=DEV) * 0.02)
        w2[e], w2_s[e] = workloads.quantize_weight_128x128(torch.randn(H, I, generator=g, device=DEV) * 0.02)
    step = [logits, bias, hs, hs_scale]
    out = torch.empty(T, H, dtype=torch.float32 if case["mode"] == "partial" else torch.bfloat16, device=DEV)
    if case["mode"] == "host":
        step = [t.cpu().pin_memory() for t in step]
        out = torch.empty(T, H, dtype=torch.bfloat16, pin_memory=True)
    if case["mode"] == "packed":
        call, weights = pkg.run_moe_prepacked, [pkg.prepack_weights(w13, w2), w13_s, w2_s]
    else:
        call, weights = (pkg.run_moe_host if case["mode"] == "host" else pkg.run_moe), [w13, w13_s, w2, w2_s]
    return call, (*step, *weights, case["offset"], 2.5, out)


def _lengths(case):
    """The batch's sequence lengths: spread evenly over the logarithm of the range."""
    n, a, b = case["batch"], case["shortest"], case["longest"]
    return [b] if n == 1 else [int(round(a * (b / a) ** (i / (n - 1)))) for i in range(n)]


def _prepare_dsa(case, seed):
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    lens = _lengths(case)
    order = torch.randperm(len(lens), generator=torch.Generator().manual_seed(int(seed))).tolist()
    lens = [lens[i] for i in order]
    need = [(n + PAGE - 1) // PAGE for n in lens]
    pages, B = sum(need) + 3, case["batch"]
    q = torch.randn(B, HEADS, DIM, generator=g, device=DEV).to(torch.float8_e4m3fn)
    keys = torch.randn(pages, PAGE, DIM, generator=g, device=DEV)
    keys *= 0.5 + torch.rand(pages, PAGE, 1, generator=g, device=DEV)
    scale = keys.abs().amax(-1, keepdim=True).clamp_min(1e-6) / 448.0
    cache = torch.empty(pages, PAGE * (DIM + 4), dtype=torch.uint8, device=DEV)
    cache[:, : PAGE * DIM] = (keys / scale).to(torch.float8_e4m3fn).view(torch.uint8).view(pages, PAGE * DIM)
    cache[:, PAGE * DIM:] = scale.view(pages, PAGE).view(torch.uint8)
    weights = torch.randn(B, HEADS, generator=g, device=DEV) / 8.0
    # every sequence's pages lie scattered over the cache
    place = torch.randperm(pages, generator=g, device=DEV).to(torch.int32)
    table = torch.zeros(B, case["table_pages"], dtype=torch.int32, device=DEV)
    at = 0
    for b, n in enumerate(need):
        table[b, :n] = place[at: at + n]
        at += n
    out = torch.empty(B, TOPK, dtype=torch.int32, device=DEV)
    return pkg.run_dsa_topk_indexer, (q, cache.view(torch.int8).view(pages, PAGE, 1, DIM + 4), weights,
                                      torch.tensor(lens, dtype=torch.int32, device=DEV), table, out)


def prepare(case, seed):
    return _prepare_dsa(case, seed) if case["op"] == "dsa" else _prepare_moe(case, seed)


def run(state):
    call, args = state
    return call(*args)


# ------------------------------------------------------------------------------------------------- what a pass needs
def _routing_counts(case):
    """(routed rows, active experts) of the local slice, from one draw of the router's inputs on the host."""
    x, bias = _logits(case, torch.Generator().manual_seed(0), "cpu")
    v = torch.sigmoid(x) + bias.float()
    groups = v.view(-1, 8, 32).topk(2, dim=-1).values.sum(-1).topk(4, dim=-1).indices
    kept = torch.zeros(len(v), 8, dtype=torch.bool).scatter_(1, groups, True).repeat_interleave(32, dim=1)
    local = v.masked_fill(~kept, -math.inf).topk(8, dim=-1).indices - case["offset"]
    local = local[(local >= 0) & (local < case["experts"])]
    return local.numel(), local.unique().numel()


def work(case):
    if case["op"] == "dsa":
        tokens = sum(_lengths(case))
        # a token's key bytes and scale, a sequence's query, head weights and result
        return {"bytes": tokens * (DIM + 4) + case["batch"] * (HEADS * DIM + HEADS * 4 + TOPK * 4) + tokens // PAGE * 4,
                "flops": tokens * HEADS * DIM * 2}
    routes, active = _routing_counts(case)
    flops, size = workloads.algorithmic_work(routes, active, case["tokens"])
    if case["mode"] == "partial":
        size += case["tokens"] * workloads.HIDDEN * 2      # f32 instead of bf16 rows
    return {"bytes": size, "flops": flops}


def tolerance(case):
    if case["op"] == "dsa":
        # whole numbers in score order; only tokens whose f32 scores agree to the last bits may change places
        return {"rel": 0.0, "differ": 2e-3}
    # the intermediate between the two GEMMs carries about eight mantissa bits, bf16 results as many
    return {"rel": 5e-3, "max": 5e-2}
