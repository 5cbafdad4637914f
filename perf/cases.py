"""The workloads this library is measured on, each one pass of its public entry points on one GPU.

A case says what a host program asks for (rows, vocabulary, options, data type, entry point); `prepare`
builds what such a program holds before the call — device-resident logits of its forward pass, the
handle, the output buffers it reuses — and `run` makes the call.  The shapes are those of the
benchmark and the tests: the five sampler configurations, the router, the regroup gather, speculative
verification and the latent-attention indexer, from a single Session's decode step to a large batch.
"""
import math
import random

import numpy as np
import torch

from __graft_entry__ import load_package

package = load_package()

DEVICE = "cuda"
HOT_SPOTS = 32      # boosted logits of a peaked row
ROUTER_SCORES = {"softmax": package.ROUTER_SOFTMAX, "sigmoid": package.ROUTER_SIGMOID, "sqrtsoftplus": package.ROUTER_SQRT_SOFTPLUS}


def listed():
    return [
        # One Session decoding alone: a single row per step, the token back on the host before the next step.
        dict(name="decode_1_row", kind="sample", entry="tokens", rows=1, vocab=201088, dtype="f32", options="topk", top_k=50),
        # A few Sessions with nucleus sampling only (no Top-K, the common API default): the whole vocabulary is ranked.
        dict(name="decode_8_rows_nucleus", kind="sample", entry="tokens", rows=8, vocab=151936, dtype="f32", options="nucleus", top_k=0),
        # The headline batch: 256 Sessions per step, resident parameters, Top-K ids listed.
        dict(name="batch_256_f32", kind="sample", entry="batch", rows=256, vocab=201088, dtype="f32", options="topk", top_k=50),
        # The same batch from a bf16 LM head.
        dict(name="batch_256_bf16", kind="sample", entry="batch", rows=256, vocab=201088, dtype="bf16", options="topk", top_k=50),
        # Greedy and plain temperature Sessions side by side, bf16.
        dict(name="greedy_and_temperature", kind="sample", entry="batch", rows=256, vocab=129280, dtype="bf16", options="temperature", top_k=0),
        # A large cross-Session batch in which every Session brings its own options.
        dict(name="mixed_1024_rows", kind="sample", entry="batch", rows=1024, vocab=151936, dtype="f32", options="mixed", top_k=0),
        # The largest batch: heavy-tailed bf16 logits, Top-P only.
        dict(name="heavy_tail_2048_rows", kind="sample", entry="batch", rows=2048, vocab=201088, dtype="bf16", options="heavy", top_k=0),
        # One rank's share of a vocabulary-sharded step: local candidates of its slice, merge of the gathered lists.
        dict(name="vocab_shard_of_8", kind="sharded", rows=64, vocab=131072, shards=8, dtype="f32", top_k=64),
        # MoE prefill: a router call over a chunk of tokens, then the regrouped activations.
        dict(name="router_prefill", kind="router", tokens=4096, experts=256, top_k=8, score="sigmoid", bias=True, columns=4096),
        # MoE decode: the same for the handful of tokens of one decode step.
        dict(name="router_decode", kind="router", tokens=32, experts=128, top_k=4, score="softmax", bias=False, columns=2880),
        # Speculative decoding: 32 Sessions verify four proposals each.
        dict(name="speculative_32_sessions", kind="speculative", sessions=32, draft=4, vocab=201088, dtype="f32", top_k=40),
        # Latent attention: the indexer picks the history entries of a chunk of query tokens.
        dict(name="indexer_64_rows", kind="indexer", rows=64, count=40000, top_k=2048),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng: random.Random):
    kind = rng.choice(["sample"] * 6 + ["sharded", "router", "router", "speculative", "indexer"])
    if kind == "sample":
        dtype = rng.choice(["f32", "bf16"])
        options = rng.choice(["topk", "topk", "nucleus", "temperature", "mixed", "heavy"])
        entry = rng.choice(["batch", "tokens"])
        vocab = _log_int(rng, 32000, 262144)
        most = 512 if options in ("nucleus", "temperature") else 1024
        rows = min(_log_int(rng, 1, most), 150_000_000 // vocab)
        return dict(kind=kind, entry=entry, rows=rows, vocab=vocab, dtype=dtype, options=options, top_k=_log_int(rng, 1, 256) if options == "topk" else 0)
    if kind == "sharded":
        return dict(kind=kind, rows=_log_int(rng, 1, 128), vocab=_log_int(rng, 16384, 524288), shards=rng.choice([2, 4, 8]), dtype=rng.choice(["f32", "bf16"]),
                    top_k=_log_int(rng, 8, 128))
    if kind == "router":
        return dict(kind=kind, tokens=_log_int(rng, 1, 4096), experts=rng.choice([32, 64, 128, 160, 256, 384]), top_k=rng.choice([2, 4, 6, 8]),
                    score=rng.choice(sorted(ROUTER_SCORES)), bias=rng.random() < 0.5, columns=rng.choice([1024, 2048, 2880, 4096]))
    if kind == "speculative":
        return dict(kind=kind, sessions=_log_int(rng, 1, 48), draft=rng.randint(1, 6), vocab=_log_int(rng, 32000, 201088), dtype=rng.choice(["f32", "bf16"]),
                    top_k=_log_int(rng, 10, 100))
    return dict(kind=kind, rows=_log_int(rng, 1, 128), count=_log_int(rng, 1024, 131072), top_k=rng.choice([512, 1024, 2048]))


# ---- inputs ----------------------------------------------------------------------------------------


def _generators(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed)), np.random.default_rng(int(seed))


def _spiked(generator, logits, low, high, count):
    rows, vocab = logits.shape
    where = torch.randint(vocab, (rows, count), generator=generator, device=DEVICE)
    boost = low + (high - low) * torch.rand((rows, count), generator=generator, device=DEVICE)
    logits.scatter_add_(1, where, boost)


def _heavy_tailed(generator, rows, vocab):
    """2 * Student-t(3) as bf16, a few rows at a time (the generator needs four normals per logit)."""
    logits = torch.empty((rows, vocab), dtype=torch.bfloat16, device=DEVICE)
    for begin in range(0, rows, 256):
        n = min(256, rows - begin)
        chi = torch.zeros((n, vocab), device=DEVICE)
        for _ in range(3):
            chi += torch.randn((n, vocab), generator=generator, device=DEVICE).square_()
        logits[begin:begin + n] = torch.randn((n, vocab), generator=generator, device=DEVICE).mul_(2.0).div_(chi.div_(3.0).sqrt_())
    return logits


def _logits(case, generator):
    rows, vocab, options = case["rows"], case["vocab"], case["options"]
    if options == "heavy":
        logits = _heavy_tailed(generator, rows, vocab)
        return logits if case["dtype"] == "bf16" else logits.float()
    sigma = 2.0 if options == "temperature" else 3.0
    logits = torch.randn((rows, vocab), generator=generator, device=DEVICE).mul_(sigma)
    if options == "topk":
        _spiked(generator, logits, 5.0, 15.0, HOT_SPOTS)
        # exact duplicates, as quantised heads produce them
        where = torch.randint(vocab, (2, rows, 64), generator=generator, device=DEVICE)
        logits.scatter_(1, where[0], logits.gather(1, where[1]))
    elif options in ("mixed", "nucleus"):
        _spiked(generator, logits, 4.0, 12.0, 16)
    if case["dtype"] == "bf16":
        logits = logits.bfloat16()
    if options == "temperature":
        # one row in ten carries a four-way tie at its maximum
        tied = torch.arange(0, rows, 10, device=DEVICE)
        where = torch.randint(vocab, (tied.numel(), 4), generator=generator, device=DEVICE)
        logits[tied[:, None], where] = logits[tied].amax(dim=1, keepdim=True)
    return logits


def _row_params(case, rng, seed):
    rows, options = case["rows"], case["options"]
    if options == "topk":
        return package.make_row_params(rows, temperature=0.7, top_k=case["top_k"], top_p=0.9, min_p=0.05, seed=seed)
    if options == "nucleus":
        return package.make_row_params(rows, temperature=rng.uniform(0.6, 1.2, rows).astype(np.float32), top_p=rng.uniform(0.85, 0.99, rows).astype(np.float32), seed=seed)
    if options == "temperature":
        return package.make_row_params(rows, temperature=np.where(np.arange(rows) % 2 == 0, 0.0, 1.0).astype(np.float32), seed=seed)
    if options == "heavy":
        return package.make_row_params(rows, temperature=1.0, top_p=0.95, seed=seed)
    return package.make_row_params(rows, temperature=rng.uniform(0.3, 1.5, rows).astype(np.float32), top_k=rng.choice(np.array([1, 20, 40, 100, 0], dtype=np.uint32), rows),
                                   top_p=rng.uniform(0.5, 1.0, rows).astype(np.float32), min_p=rng.choice(np.array([0.0, 0.02, 0.1], dtype=np.float32), rows), seed=seed)


def _prepare_sample(case, seed):
    generator, rng = _generators(seed)
    rows = case["rows"]
    state = dict(case=case, logits=_logits(case, generator), params=_row_params(case, rng, seed), step=0,
                 sampler=package.Sampler(max_rows=rows, max_vocab=case["vocab"]))
    if case["entry"] == "tokens":
        # page-locked results, so that the copy back needs no staging
        pinned = torch.empty(rows * package.SAMPLED_ROW_DTYPE.itemsize, dtype=torch.uint8, pin_memory=True)
        state["pinned"] = pinned
        state["results"] = pinned.numpy().view(package.SAMPLED_ROW_DTYPE)
    else:
        top_k = case["top_k"]
        state["out"] = {name: torch.empty(rows, dtype=dtype, device=DEVICE)
                        for name, dtype in (("token", torch.int32), ("probability", torch.float32), ("flags", torch.int32), ("status", torch.int32))}
        state["out"]["topk"] = torch.empty((rows, top_k), dtype=torch.int32, device=DEVICE) if top_k else None
    return state


def _rank_records(values, first_index):
    """The best-first 64-bit candidate records (ordered logit bits, inverted token id) of a [rows, n] matrix and its ids."""
    bits = values.view(torch.int32).to(torch.int64) & 0xFFFFFFFF
    key = torch.where(bits >= 0x80000000, bits ^ 0xFFFFFFFF, bits | 0x80000000)
    records = (key << 32) | (0xFFFFFFFF - first_index)
    return records.sort(dim=1, descending=True).values   # the best logits are positive: one sign bit, so signed order is record order


def _prepare_sharded(case, seed):
    generator, _ = _generators(seed)
    rows, vocab, shards, top_k = case["rows"], case["vocab"], case["shards"], case["top_k"]
    own = shards // 2
    gathered = torch.empty((shards, rows, top_k), dtype=torch.int64, device=DEVICE)
    logits = None
    for shard in range(shards):
        part = torch.randn((rows, vocab), generator=generator, device=DEVICE).mul_(3.0)
        if case["dtype"] == "bf16":
            part = part.bfloat16()
        if shard == own:
            logits = part
        else:
            values, index = part.float().topk(top_k, dim=1)
            gathered[shard] = _rank_records(values, index + shard * vocab)
    params = package.make_row_params(rows, temperature=1.0, top_k=top_k, top_p=0.9, seed=seed)
    out = {name: torch.empty(rows, dtype=dtype, device=DEVICE)
           for name, dtype in (("token", torch.int32), ("probability", torch.float32), ("flags", torch.int32), ("status", torch.int32))}
    out["topk"] = torch.empty((rows, top_k), dtype=torch.int32, device=DEVICE)
    return dict(case=case, logits=logits, gathered=gathered, own=own, params=params, out=out, step=0, sampler=package.Sampler(max_rows=rows, max_vocab=vocab))


def _prepare_router(case, seed):
    generator, _ = _generators(seed)
    tokens, experts = case["tokens"], case["experts"]
    logits = torch.randn((tokens, experts), generator=generator, device=DEVICE)
    bias = torch.randn(experts, generator=generator, device=DEVICE).mul_(0.1) if case["bias"] else None
    hidden = torch.randn((tokens, case["columns"]), generator=generator, device=DEVICE)
    routes = tokens * case["top_k"]
    plan = package.DispatchPlan(torch.empty(experts + 1, dtype=torch.int32, device=DEVICE), torch.empty(routes, dtype=torch.int32, device=DEVICE),
                                torch.empty(routes, dtype=torch.int32, device=DEVICE), torch.empty(routes, dtype=torch.float32, device=DEVICE),
                                torch.zeros(1, dtype=torch.int32, device=DEVICE))
    return dict(case=case, logits=logits, bias=bias, hidden=hidden, plan=plan, sampler=package.Sampler(max_rows=1, max_vocab=1))


def _prepare_speculative(case, seed):
    generator, rng = _generators(seed)
    sessions, draft_count, vocab, top_k = case["sessions"], case["draft"], case["vocab"], case["top_k"]
    target = torch.randn((sessions, draft_count + 1, vocab), generator=generator, device=DEVICE).mul_(2.5)
    # draft models of every quality, from nearly the target to a poor guess
    closeness = torch.tensor(np.exp(rng.uniform(math.log(0.05), math.log(1.2), sessions)).astype(np.float32), device=DEVICE)[:, None, None]
    draft = target[:, :draft_count] + closeness * torch.randn((sessions, draft_count, vocab), generator=generator, device=DEVICE)
    if case["dtype"] == "bf16":
        target, draft = target.bfloat16(), draft.bfloat16()
    # the draft model's own samples: a draw among its best candidates, well inside its nucleus
    values, index = draft.float().topk(min(top_k, 16), dim=2)
    weights = torch.softmax(values, dim=2)
    weights[..., 1:] *= (weights.cumsum(dim=2)[..., :-1] < 0.8)
    pick = torch.multinomial(weights.view(sessions * draft_count, -1), 1, generator=generator).view(sessions, draft_count, 1)
    proposed = index.gather(2, pick).squeeze(2).to(torch.int32).contiguous()
    params = package.make_row_params(sessions, temperature=1.0, top_k=top_k, top_p=0.95, seed=seed)
    out = (torch.zeros(sessions * draft_count, dtype=torch.float32, device=DEVICE),
           torch.zeros(sessions * package.SPECULATIVE_RESULT_DTYPE.itemsize, dtype=torch.uint8, device=DEVICE))
    return dict(case=case, target=target, draft=draft, proposed=proposed, params=params, out=out,
                sampler=package.Sampler(max_rows=sessions * (2 * draft_count + 1), max_vocab=vocab))


def _prepare_indexer(case, seed):
    generator, _ = _generators(seed)
    shape = (case["rows"], case["count"])
    # sums of relu(dot) * weight: many exact zeros, a few large values
    scores = torch.randn(shape, generator=generator, device=DEVICE).clamp_(min=0.0).mul_(torch.rand(shape, generator=generator, device=DEVICE))
    return dict(case=case, scores=scores, sampler=package.Sampler(max_rows=1, max_vocab=1))


def prepare(case, seed):
    return {"sample": _prepare_sample, "sharded": _prepare_sharded, "router": _prepare_router, "speculative": _prepare_speculative,
            "indexer": _prepare_indexer}[case["kind"]](case, seed)


# ---- one pass --------------------------------------------------------------------------------------


def run(state):
    case, sampler = state["case"], state["sampler"]
    kind = case["kind"]
    if kind == "sample":
        # the parameters go up with the first step and stay resident; later steps only advance the counter
        params = state["params"] if state["step"] == 0 else None
        step, state["step"] = state["step"], state["step"] + 1
        if case["entry"] == "tokens":
            results = sampler.sample_tokens(state["logits"], params, step_offset=step, results=state["results"])
            return {name: results[name] for name in package.SAMPLED_ROW_DTYPE.names}
        return sampler.sample_batch(state["logits"], params, step_offset=step, topk_stride=case["top_k"], out=state["out"])
    if kind == "sharded":
        params = state["params"] if state["step"] == 0 else None
        step, state["step"] = state["step"], state["step"] + 1
        sampler.local_candidates(state["logits"], state["own"] * case["vocab"], case["top_k"], out=state["gathered"][state["own"]])
        out = sampler.merge_candidates(state["gathered"], params, case["top_k"], step_offset=step, topk_stride=case["top_k"], out=state["out"])
        return {"candidates": state["gathered"], **out}
    if kind == "router":
        plan = sampler.router_dispatch(state["logits"], case["top_k"], score_function=ROUTER_SCORES[case["score"]], selection_bias=state["bias"], out=state["plan"])
        gathered = sampler.regroup_gather(state["hidden"], plan.route_token)
        return {"offsets": plan.expert_offsets, "token": plan.route_token, "rank": plan.route_rank, "weight": plan.route_weight, "status": plan.status,
                "gathered": gathered}
    if kind == "speculative":
        return sampler.speculative_verify_batch(state["target"], state["draft"], state["proposed"], state["params"], out=state["out"], sync=False)
    return sampler.indexer_topk(state["scores"], case["top_k"], with_scores=True)


def work(case):
    """Bytes every pass has to move (inputs read once, outputs written once) and the arithmetic it cannot do without."""
    kind = case["kind"]
    size = 4 if case.get("dtype", "f32") == "f32" else 2
    if kind == "sample":
        logits = case["rows"] * case["vocab"]
        # a comparison per logit; a row ranked without Top-K also needs its exponential and one sum
        per_logit = {"topk": 1, "mixed": 2, "heavy": 4, "nucleus": 4, "temperature": 3}[case["options"]]
        return {"bytes": logits * size + case["rows"] * (40 + 16 + 4 * case["top_k"]), "flops": logits * per_logit}
    if kind == "sharded":
        logits = case["rows"] * case["vocab"]
        return {"bytes": logits * size + case["rows"] * (case["top_k"] * (8 * case["shards"] + 8 + 4) + 40 + 16), "flops": logits}
    if kind == "router":
        routes = case["tokens"] * case["top_k"]
        hidden = case["tokens"] * case["columns"] * 4
        return {"bytes": case["tokens"] * case["experts"] * 4 + routes * 12 + case["experts"] * 8 + hidden + routes * case["columns"] * 4,
                "flops": case["tokens"] * case["experts"] * 4}
    if kind == "speculative":
        logits = case["sessions"] * (2 * case["draft"] + 1) * case["vocab"]
        return {"bytes": logits * size + case["sessions"] * (64 + 8 * case["draft"]), "flops": logits}
    logits = case["rows"] * case["count"]
    return {"bytes": logits * 4 + case["rows"] * case["top_k"] * 8, "flops": logits}


def tolerance(case):
    # Token ids, Top-K lists, routes, regrouped rows and the indexer's choice are whole values or copies: the
    # reference's sequential sums are replayed, so they do not move.  Probabilities and weights are quotients of such
    # sums; a correctly rounded exp and the host library's differ by one unit in the last place for a few arguments in ten
    # thousand, which moves a probability by about 1e-7.
    if case["kind"] == "indexer":
        return "exact"
    return {"rel": 5e-7, "max": 2e-6, "differ": 0.0}
