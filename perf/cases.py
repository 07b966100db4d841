"""Performance cases: the work that a serving engine hands to this library.

Every case is one pass through the public entry points (`pagoda_b200.Sampler`): a decode step over a batch of rows, the
scoring of candidate continuations, or one rank's share of a vocabulary-sharded step.  Inputs follow the recipes of
`pagoda_b200.synth` (normal logits, a few spiked tokens per row, uniform history ids, random grammar masks), made on the
GPU from the seed.
"""
import math

import numpy as np
import torch

import pagoda_b200

V = 151936          # the vocabulary that the benchmark is quoted on
V_LARGE = 256000    # the largest vocabulary among the benchmark configurations
LARGEST = 256 * V   # logits of the largest listed batch

# Fields of a decode step that a case may leave out: one value for every row, as a single-tenant server sends them.
STEP = dict(kind="step", dtype="f32", temperature=0.7, top_k=50, top_p=0.9, freq=0.0, pres=0.0, rep=1.0, history=0,
            states=0, masked=0.0, greedy_share=0.0, mixed=False, exact=False)


def listed():
    return [
        # One chat, greedy with a repetition penalty over the text so far: the smallest call, latency alone.
        dict(STEP, name="greedy_b1", rows=1, vocab=V, temperature=0.0, top_k=0, top_p=1.0, rep=1.1, history=112),
        # A handful of chats with the usual sampling settings: an interactive server at low load.
        dict(STEP, name="chat_b8", rows=8, vocab=V, temperature=0.8, top_k=40, top_p=0.95, freq=0.2, pres=0.1, history=256),
        # An ordinary batch of the continuous batcher, penalties over half a thousand ids.
        dict(STEP, name="topk_topp_b64", rows=64, vocab=V, freq=0.2, pres=0.1, history=512),
        # Constrained decoding: every row under a grammar mask, half of them greedy (tool calls), half sampled.
        dict(STEP, name="grammar_b128", rows=128, vocab=V, temperature=1.0, top_k=20, top_p=1.0, states=64, masked=1.0,
             greedy_share=0.5),
        # The headline batch: a full decode step of a throughput server.
        dict(STEP, name="headline_b256", rows=256, vocab=V, freq=0.2, pres=0.1, history=512),
        # Many tenants in one batch: bf16 logits, every row its own parameters, long histories, some rows constrained.
        dict(STEP, name="hetero_bf16_b256", rows=256, vocab=V_LARGE, dtype="bf16", mixed=True, history=2048, states=4,
             masked=0.3),
        # The parameters' defaults: top-k off, half of the rows with top-p off too (plain categorical draw), half nucleus.
        dict(STEP, name="open_b32", rows=32, vocab=V, temperature=0.7, top_k=0, top_p=0.95, freq=0.2, pres=0.1, history=256),
        # A vocabulary that is no multiple of anything, rows packed without padding.
        dict(STEP, name="ragged_b48", rows=48, vocab=50257, temperature=0.8, top_k=40, top_p=0.95, rep=1.1, history=200),
        # The bit-exact mode, for runs that have to be reproduced token by token.
        dict(STEP, name="exact_b16", rows=16, vocab=V, freq=0.2, pres=0.1, history=512, exact=True),
        # Scoring candidate continuations: the log-probability of one id per position.
        dict(name="score_b64", kind="score", rows=64, vocab=V, full=False),
        # One rank of an eight-way vocabulary split with four-token draft verification: emit, merge, accept.
        dict(name="shard_b1024", kind="shard", rows=1024, vocab=V, shards=8, cand=64, positions=4, top_p=0.95),
        # Logits in pinned host memory, tokens back on the host: an engine whose model does not run on this GPU.
        dict(STEP, name="host_b32", kind="host", rows=32, vocab=V, freq=0.2, pres=0.1, history=512),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["greedy", "sample", "sample", "grammar", "hetero", "open", "exact", "score", "shard", "host"])
    vocab = _log_int(rng, 1000, V_LARGE)
    vocab -= vocab % rng.choice([1, 2, 8, 64, 128])
    most = {"open": 32, "exact": 32, "host": 32, "score": 64, "shard": 1024}.get(kind, 256)
    rows = _log_int(rng, 4 if kind == "shard" else 1, most)
    rows = max(1, min(rows, LARGEST // vocab))
    step = dict(STEP, rows=rows, vocab=vocab, dtype=rng.choice(["f32", "f32", "bf16"]), temperature=round(rng.uniform(0.5, 1.2), 3),
                top_k=_log_int(rng, 1, min(1024, vocab - 1)), top_p=rng.choice([1.0, round(rng.uniform(0.5, 0.99), 3)]))
    if rng.random() < 0.6:
        step.update(history=_log_int(rng, 16, 2048), freq=rng.choice([0.0, 0.2]), pres=rng.choice([0.0, 0.1]), rep=rng.choice([1.0, 1.1]))
    if kind == "greedy":
        step.update(temperature=0.0, top_k=0, top_p=1.0)
    elif kind == "grammar":
        step.update(states=rng.randint(2, 64), masked=rng.choice([0.5, 1.0]), greedy_share=rng.choice([0.0, 0.5]))
    elif kind == "hetero":
        step.update(mixed=True, states=4, masked=0.3)
    elif kind == "open":
        step.update(top_k=0)
    elif kind == "exact":
        step.update(exact=True)
    elif kind == "host":
        step.update(kind="host", dtype="f32")
    elif kind == "score":
        return dict(kind="score", rows=rows, vocab=vocab, full=rng.random() < 0.25)
    elif kind == "shard":
        shards = rng.choice([2, 4, 8])
        vocab = max(64 * shards, min(vocab, V * shards // 8))   # a rank's columns are no wider than in the listed case
        vocab -= vocab % (4 * shards)
        positions = rng.choice([1, 2, 4])
        return dict(kind="shard", rows=max(1, rows // positions) * positions, vocab=vocab, shards=shards,
                    cand=rng.choice([16, 32, 64]), positions=positions, top_p=rng.choice([0.9, 0.95, 1.0]))
    return step


# ------------------------------------------------------------------------------------------------ inputs

def _logits(gen, rows, vocab, std=2.0, spikes=8):
    """Normal logits with a few tokens per row lifted by 10, as a language model's head produces them."""
    dev = gen.device
    x = torch.randn(rows, vocab, generator=gen, device=dev) * std
    if spikes:
        ids = torch.randint(0, vocab, (rows, spikes), generator=gen, device=dev)
        x.scatter_add_(1, ids, torch.full((rows, spikes), 10.0, device=dev))
    return x


def _mask_table(gen, states, vocab, lo, hi):
    """One bitmask per grammar state, 32 tokens to the word, token 0 always allowed."""
    dev = gen.device
    words = (vocab + 31) // 32
    density = lo + (hi - lo) * torch.rand(states, 1, generator=gen, device=dev)
    bits = torch.rand(states, words * 32, generator=gen, device=dev) < density
    bits[:, 0] = True
    bits[:, vocab:] = False
    weights = 1 << torch.arange(32, device=dev, dtype=torch.int64)
    packed = (bits.view(states, words, 32).to(torch.int64) * weights).sum(2)
    return packed.cpu().numpy().astype(np.uint32)


def _step_rows(case, gen):
    """Per-row parameters of a decode step, on the GPU."""
    dev, rows, vocab = gen.device, case["rows"], case["vocab"]

    def rand(lo, hi):
        return lo + (hi - lo) * torch.rand(rows, generator=gen, device=dev)

    def full(v, dt=torch.float32):
        return torch.full((rows,), v, dtype=dt, device=dev)

    p = dict(temperature=full(case["temperature"]), top_k=full(case["top_k"], torch.int32), top_p=full(case["top_p"]),
             frequency_penalty=full(case["freq"]), presence_penalty=full(case["pres"]), repetition_penalty=full(case["rep"]))
    if case["mixed"]:
        p.update(temperature=rand(0.3, 1.5), top_k=rand(1, min(1024, vocab - 1)).to(torch.int32), top_p=rand(0.5, 1.0),
                 repetition_penalty=rand(1.0, 1.3))
    elif case["top_k"] == 0 and case["temperature"] > 0:
        p["top_p"][::2] = 1.0
    greedy = int(rows * case["greedy_share"])
    if greedy:
        p["temperature"][:greedy] = 0.0
        p["top_k"][:greedy] = 0
    if case["history"]:
        p["hist_offsets"] = torch.arange(rows + 1, dtype=torch.int32, device=dev) * case["history"]
        p["hist_ids"] = torch.randint(0, vocab, (rows * case["history"],), generator=gen, dtype=torch.int32, device=dev)
    p["uniform"] = torch.rand(rows, generator=gen, device=dev)
    return p


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    rows, vocab = case["rows"], case["vocab"]
    if case["kind"] == "score":
        s = pagoda_b200.Sampler(device=dev.index, max_rows=rows, max_vocab=vocab, max_history=1)
        ids = torch.randint(0, vocab, (rows,), generator=gen, dtype=torch.int32, device=dev)
        return dict(case=case, sampler=s, logits=_logits(gen, rows, vocab), ids=ids)
    if case["kind"] == "shard":
        return _prepare_shard(case, gen)

    s = pagoda_b200.Sampler(device=dev.index, max_rows=rows, max_vocab=vocab, max_history=max(1, case["history"]))
    s.set_exact(case["exact"])
    x = _logits(gen, rows, vocab, 2.5 if case["mixed"] else 2.0, 0 if case["mixed"] or case["states"] else 8)
    p = _step_rows(case, gen)
    if case["kind"] == "host":
        p = {k: v.cpu().numpy() for k, v in p.items()}
        pinned = x.cpu().pin_memory()
        return dict(case=case, sampler=s, pinned=pinned, logits=pinned.numpy(), params=p)

    if case["states"]:
        lo, hi = (0.05, 0.05) if case["mixed"] else (0.01, 0.20)
        table = s.upload_mask_table(_mask_table(gen, case["states"], vocab, lo, hi))
        masked = torch.rand(rows, generator=gen, device=dev) < case["masked"]
        p["mask_table"] = torch.where(masked, table, -1).to(torch.int32)
        p["mask_state"] = torch.randint(0, case["states"], (rows,), generator=gen, dtype=torch.int32, device=dev)
    out = dict(token=torch.zeros(rows, dtype=torch.int32, device=dev), status=torch.zeros(rows, dtype=torch.int32, device=dev),
               drew=torch.zeros(rows, dtype=torch.uint8, device=dev), argmax=torch.zeros(rows, dtype=torch.int32, device=dev),
               row_max=torch.zeros(rows, device=dev), sumexp=torch.zeros(rows, device=dev), total=torch.zeros(rows, device=dev))
    if case["top_k"]:   # (rows over the whole vocabulary: no server asks how many entries they keep)
        out["n_kept"] = torch.zeros(rows, dtype=torch.int32, device=dev)
    desc = s.make_device_desc(x.to(torch.bfloat16) if case["dtype"] == "bf16" else x, **out, **p)
    return dict(case=case, sampler=s, desc=desc, out=out)


def _prepare_shard(case, gen):
    """Rank 0's columns, and the records of the other ranks as the all-gather delivers them."""
    dev, rows, n, cand = gen.device, case["rows"], case["shards"], case["cand"]
    width = case["vocab"] // n
    s = pagoda_b200.Sampler(device=dev.index, max_rows=rows, max_vocab=width, max_history=16)
    t = torch.ones(rows, device=dev)
    records = torch.zeros((n, rows, s.tp_record_bytes(cand)), dtype=torch.uint8, device=dev)
    stream = torch.cuda.current_stream().cuda_stream
    for r in range(n - 1, -1, -1):
        x = _logits(gen, rows, width, spikes=0)
        s.tp_partial(x, case["vocab"], n, r, cand, temperature=t, records=records[r], stream_ptr=stream)
    seqs = rows // case["positions"]
    # drafts that agree with the model about half of the time
    head = records.view(torch.int32)[:, :, 3]
    best = records.view(torch.float32)[:, :, 0].argmax(0, keepdim=True)
    am = head.gather(0, best)[0]
    miss = torch.rand(rows, generator=gen, device=dev) < 0.25
    draft = torch.where(miss, torch.randint(0, case["vocab"], (rows,), generator=gen, dtype=torch.int32, device=dev), am)
    zeros = lambda: torch.zeros(seqs, dtype=torch.int32, device=dev)  # noqa: E731
    return dict(case=case, sampler=s, shard=x, records=records, temperature=t, top_p=torch.full((rows,), case["top_p"], device=dev),
                uniform=torch.rand(rows, generator=gen, device=dev), draft=draft.view(seqs, -1).contiguous(),
                out=s.tp_outputs(rows, dev), accept=(zeros(), zeros()))


# ------------------------------------------------------------------------------------------------ one pass

def run(state):
    case, s = state["case"], state["sampler"]
    if case["kind"] == "host":
        r = s.sample_batch(state["logits"], diagnostics=True, **state["params"])
        return dict(token=r.token.astype(np.int64), status=r.status, drew=r.drew, argmax=r.argmax.astype(np.int64),
                    row_max=r.row_max, sumexp=r.sumexp, total=r.total, n_kept=r.n_kept.astype(np.int64))
    stream = torch.cuda.current_stream().cuda_stream
    if case["kind"] == "step":
        s.launch_device(state["desc"], stream)
        return state["out"]
    if case["kind"] == "score":
        gathered, full, status = s.log_softmax(state["logits"], ids=state["ids"], full=case["full"], stream_ptr=stream)
        return dict(gathered=gathered, full=full, status=status)
    n, cand, vocab = case["shards"], case["cand"], case["vocab"]
    rec = state["records"]
    s.tp_partial(state["shard"], vocab, n, 0, cand, temperature=state["temperature"], records=rec[0], stream_ptr=stream)
    out = s.tp_merge(rec, vocab, n, 0, cand, temperature=state["temperature"], top_p=state["top_p"], uniform=state["uniform"],
                     stream_ptr=stream, out=state["out"])
    draft = state["draft"]
    accepted, following = s.draft_accept(out["argmax"].view(draft.shape), draft, stream_ptr=stream, out=state["accept"])
    f, i = rec[0].view(torch.float32), rec[0].view(torch.int32)
    return dict(out, accepted=accepted, following=following, shard_max=f[:, 0], shard_sum=f[:, 1], shard_status=i[:, 2],
                shard_argmax=i[:, 3], shard_logits=f[:, 4:4 + cand], shard_ids=i[:, 4 + cand:4 + 2 * cand])


def work(case):
    rows, vocab = case["rows"], case["vocab"]
    if case["kind"] == "score":   # maximum, exponential, sum
        return dict(bytes=rows * (4 * vocab * (2 if case["full"] else 1) + 12), flops=4 * rows * vocab)
    if case["kind"] == "shard":
        record = 16 + 8 * case["cand"]
        width = vocab // case["shards"]
        return dict(bytes=rows * (4 * width + record * case["shards"] + 64), flops=4 * rows * width)
    esize = 2 if case["dtype"] == "bf16" else 4
    b = rows * (vocab * esize + 64 + 4 * case["history"]) + int(rows * case["masked"]) * (vocab // 8)
    stochastic = 0.0 if case["temperature"] == 0 else 1.0 - case["greedy_share"]
    return dict(bytes=b, flops=rows * vocab * (1 + 3 * stochastic))


def tolerance(case):
    if case["kind"] == "score":   # f32 logarithms of magnitude ten
        return dict(rel=1e-6, max=1e-6)
    if case["kind"] in ("step", "host"):
        # bit-exact mode, greedy rows, and rows over the whole vocabulary: every token depends on the exact f32 sum
        if case["exact"] or case["temperature"] == 0 or case["top_k"] == 0:
            return "exact"
    # the f32 left-fold sum within 1e-5; a draw or a top-p cut that sits that close to its boundary may go either way
    return dict(rel=1e-5, max=2e-5, differ=0.01)
