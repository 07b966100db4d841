"""The wide kernel (exact mode, unaligned rows, wide-open rows, scoring) against the oracle, at the edges of its
512-logit regions, of its row chunk, of the candidate list that one CTA finishes and of the history it takes."""
import numpy as np
import pytest

from .util import assert_same, run_both

pytestmark = pytest.mark.gpu


def check_scores(oracle, x, ids, g, full):
    g, full = g.cpu().numpy(), full.cpu().numpy()
    for r in range(len(x)):
        want = oracle.log_softmax(x[r])
        np.testing.assert_allclose(full[r], want, rtol=0, atol=1e-6 * max(1.0, np.abs(want).max()))
        assert g[r] == full[r][ids[r]]


@pytest.mark.parametrize("rows, vocab, top_k, history", [
    (1, 511, 0, 0), (70, 512, 40, 64), (65, 513, 0, 2048), (5, 1025, 1025, 2049), (9, 33025, 0, 300), (6, 70001, 2049, 300),
    (2, 1 << 20, 0, 8)])
def test_wide_kernel_edges(oracle, rows, vocab, top_k, history):
    import torch
    import pagoda_b200
    from pagoda_b200 import synth
    x = synth.normal_f32(7 + vocab, rows * vocab, 2.0).reshape(rows, vocab)
    x[:, vocab // 2] = x[:, 0]                     # ties
    w = synth.Workload(
        "wide", x, np.resize(np.float32([0.7, 1.3, 5.0]), rows), np.full(rows, top_k, np.uint32),
        np.resize(np.float32([0.95, 1.0, 0.999, 0.3]), rows), np.full(rows, 0.2, np.float32), np.full(rows, 0.1, np.float32),
        np.full(rows, 1.1, np.float32), np.arange(rows + 1, dtype=np.uint32) * history if history else None,
        np.random.default_rng(vocab).integers(0, vocab, rows * history).astype(np.uint32) if history else None,
        synth.uniform_f32(3, rows))
    s = pagoda_b200.Sampler(device=0, max_rows=rows, max_vocab=vocab, max_history=max(history, 1))
    try:
        s.set_exact(True)
        assert_same(*run_both(s, oracle, w), w)
        ids = np.arange(rows, dtype=np.int32) * (vocab - 1) // max(rows - 1, 1)
        g, full, status = s.log_softmax(torch.from_numpy(x).cuda(), ids=torch.from_numpy(ids).cuda(), full=True,
                                        stream_ptr=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert (status.cpu().numpy() == 0).all()
        check_scores(oracle, x, ids, g, full)
    finally:
        s.close()


@pytest.mark.parametrize("vocab", [512 * 33, 512 * 40 + 3])
@pytest.mark.parametrize("top_k", [0, 40])
@pytest.mark.parametrize("route", ["1", "3"])
def test_fold_changes_binade(oracle, monkeypatch, vocab, top_k, route):
    """The exact fold where its running value changes binade often, in one run of terms, at the edge of a region, or not
    at all, and where terms end on half an ulp: bit-exact sums, totals, tokens and scores."""
    import torch
    import pagoda_b200
    from pagoda_b200 import synth
    monkeypatch.setenv("PGS_WIDE_ROUTE", route)   # on the grid, or one CTA per row, whatever is quicker
    i = np.arange(vocab)
    rng = np.random.default_rng(vocab)
    noise = rng.standard_normal(vocab)
    rows = [np.zeros(vocab),                                        # one ulp pattern throughout
            -40.0 + 40.0 * i / vocab, -40.0 * i / vocab,            # rising: a new binade every few hundred terms; falling
            -0.6931472 * (i % 24), -0.6931472 * rng.integers(0, 12, vocab),   # powers of two, nearly: ties
            np.where(i < vocab // 2, -85.0, noise),                 # next to nothing, then everything
            np.where(i % 512 == 511, 4.0, -3.0) + noise, np.where(i % 512 == 0, 4.0, -3.0) + noise,   # at the regions' edges
            np.where(i == 777, 20.0, noise), 2.0 * noise]
    x = np.stack(rows).astype(np.float32) + np.float32(0.0)   # (no -0.0: the kernels report a maximum of zero as +0.0)
    n = len(x)
    w = synth.Workload("binades", x, np.resize(np.float32([1.0, 0.7]), n), np.full(n, top_k, np.uint32), np.resize(np.float32([1.0, 0.97, 0.9]), n),
                       np.zeros(n, np.float32), np.zeros(n, np.float32), np.ones(n, np.float32), None, None, synth.uniform_f32(5, n))
    s = pagoda_b200.Sampler(device=0, max_rows=n, max_vocab=vocab, max_history=1)
    try:
        s.set_exact(True)
        assert_same(*run_both(s, oracle, w), w)
        ids = np.full(n, vocab - 1, np.int32)
        g, full, _ = s.log_softmax(torch.from_numpy(x).cuda(), ids=torch.from_numpy(ids).cuda(), full=True,
                                   stream_ptr=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        check_scores(oracle, x, ids, g, full)
    finally:
        s.close()


@pytest.mark.parametrize("route", ["1", "3"])
@pytest.mark.parametrize("top_k", [0, 40])
@pytest.mark.parametrize("bf16", [False, True])
def test_terms_and_entries_share_the_staging_buffer(oracle, monkeypatch, route, top_k, bf16):
    """Rows of which most regions are added term by term, with history entries in every region and no mask: a warp stages one
    region's terms and the next region's entries in the same buffer.  Bit-exact sums, totals and tokens."""
    import pagoda_b200
    from pagoda_b200 import synth
    monkeypatch.setenv("PGS_WIDE_ROUTE", route)
    n, vocab = 8, 512 * 128
    i = np.arange(vocab)
    rng = np.random.default_rng(3)
    rows = [-40.0 + 40.0 * i / vocab, -0.6931472 * (i % 24), -0.6931472 * rng.integers(0, 12, vocab), 2.0 * rng.standard_normal(vocab)]
    x = np.stack(rows * 2).astype(np.float32) + np.float32(0.0)
    if bf16:
        x = synth.f32_to_bf16_bits(x).reshape(x.shape)
    ids = np.stack([rng.permutation(np.arange(0, vocab, 512)[:, None] + rng.integers(0, 512, (vocab // 512, 16)), axis=1).ravel()
                    for _ in range(n)]).astype(np.uint32)   # sixteen in every region
    w = synth.Workload("staged", x, np.resize(np.float32([1.0, 0.7]), n), np.full(n, top_k, np.uint32),
                       np.resize(np.float32([1.0, 0.97]), n), np.full(n, 0.2, np.float32), np.full(n, 0.1, np.float32),
                       np.full(n, 1.1, np.float32), np.arange(n + 1, dtype=np.uint32) * ids.shape[1], ids.ravel(), synth.uniform_f32(5, n))
    s = pagoda_b200.Sampler(device=0, max_rows=n, max_vocab=vocab, max_history=ids.shape[1])
    try:
        s.set_exact(True)
        assert_same(*run_both(s, oracle, w), w)
    finally:
        s.close()


@pytest.mark.parametrize("rows, vocab, top_k, history", [(1, 511, 0, 0), (160, 512, 40, 64), (149, 513, 0, 300), (5, 1025, 1025, 2049), (150, 9001, 30, 300),
                                                         (9, 33025, 0, 300), (3, 70001, 2049, 2100)])
def test_one_cta_per_row(oracle, monkeypatch, rows, vocab, top_k, history):
    """The wide kernel with one CTA per row: one row, more rows than SMs, rows that go on to the general kernel's code
    (more history than the workspace holds), short and long lists, a mask that leaves regions empty; steps and scores.  (In the
    default mode the unaligned batches take this way too, the aligned one the streaming kernel: test_listed_rows has what is listed.)"""
    import torch
    import pagoda_b200
    from pagoda_b200 import synth
    monkeypatch.setenv("PGS_WIDE_ROUTE", "3")
    x = synth.normal_f32(11 + vocab, rows * vocab, 2.0).reshape(rows, vocab)
    rng = np.random.default_rng(vocab)
    words = np.full((2, (vocab + 31) // 32), 0xffffffff, np.uint32)
    words[1, :words.shape[1] // 2] = 0
    words[1, 0] = 1
    w = synth.Workload(
        "rows", x, np.resize(np.float32([0.7, 0.0, 1.3, 5.0]), rows), np.full(rows, top_k, np.uint32), np.resize(np.float32([0.95, 1.0, 0.3]), rows),
        np.full(rows, 0.2, np.float32), np.full(rows, 0.1, np.float32), np.full(rows, 1.1, np.float32),
        np.arange(rows + 1, dtype=np.uint32) * history if history else None,
        rng.integers(0, vocab, rows * history).astype(np.uint32) if history else None, synth.uniform_f32(4, rows),
        mask_words=words, state_flags=np.zeros(2, np.uint32), mask_state=np.resize(np.int32([-1, 0, 1, -1, 1]), rows))
    s = pagoda_b200.Sampler(device=0, max_rows=rows, max_vocab=vocab, max_history=max(history, 1))
    try:
        for exact in (True, False, True):   # (on what the one before has left)
            s.set_exact(exact)
            assert_same(*run_both(s, oracle, w), w, exact=exact or vocab % 4 != 0, min_clear=0.0)   # (unaligned rows are bit-exact)
        ids = np.arange(rows, dtype=np.int32) % vocab
        g, full, _ = s.log_softmax(torch.from_numpy(x).cuda(), ids=torch.from_numpy(ids).cuda(), full=True,
                                   stream_ptr=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        check_scores(oracle, x, ids, g, full)
    finally:
        s.close()


def _mixed_rows(rows, vocab, top_k, history, greedy, seed=29):
    from pagoda_b200 import synth
    x = synth.normal_f32(seed + vocab, rows * vocab, 2.0).reshape(rows, vocab)
    return synth.Workload(
        "short rows", x, np.resize(np.float32([0.0] if greedy else [0.7, 1.3, 5.0]), rows), np.full(rows, top_k, np.uint32),
        np.resize(np.float32([0.95, 1.0, 0.3]), rows), np.full(rows, 0.2, np.float32), np.full(rows, 0.1, np.float32), np.full(rows, 1.1, np.float32),
        np.arange(rows + 1, dtype=np.uint32) * history if history else None,
        np.random.default_rng(vocab).integers(0, vocab, rows * history).astype(np.uint32) if history else None, synth.uniform_f32(4, rows))


# Many short rows: one launch that does them one way or the other; where histories may be long, two.
@pytest.mark.parametrize("max_history", [64, 2049])
@pytest.mark.parametrize("rows, vocab", [(75, 2049), (148, 2051), (149, 4096), (200, 16383), (330, 2052)])
@pytest.mark.parametrize("top_k, greedy", [(0, True), (3, False), (200, False), (0, False)])
def test_many_short_exact_rows(oracle, rows, vocab, top_k, greedy, max_history):
    import pagoda_b200
    w = _mixed_rows(rows, vocab, top_k, 40, greedy)
    w.logits[1, vocab - 1] = np.nan
    s = pagoda_b200.Sampler(device=0, max_rows=rows, max_vocab=vocab, max_history=max_history)
    try:
        s.set_exact(True)
        for _ in range(2):   # (on what the one before has left)
            assert_same(*run_both(s, oracle, w), w)
    finally:
        s.close()


# Aligned rows that the streaming kernel lists for what they ask for: more than SMs, more than are resident, rows that go on to
# the general kernel's code, and so few and short that they are done by it at once.
@pytest.mark.parametrize("rows, vocab, top_k, history", [
    (160, 9000, 0, 0), (320, 2048, 0, 30), (5, 1028, 0, 2049), (40, 4096, 1025, 2100), (1, 1028, 0, 0), (2, 1060, 0, 5), (2, 1796, 0, 0), (3, 1100, 0, 0)])
def test_listed_rows(oracle, rows, vocab, top_k, history):
    import pagoda_b200
    w = _mixed_rows(rows, vocab, top_k, history, False)
    some = _mixed_rows(rows, vocab, 40, 0, False)   # nothing to list in between
    s = pagoda_b200.Sampler(device=0, max_rows=rows, max_vocab=vocab, max_history=max(history, 1))
    try:
        for _ in range(2):
            got, want = run_both(s, oracle, w)
            assert_same(got, want, w)   # listed rows are bit-exact in the default mode too
            assert_same(*run_both(s, oracle, some), some, exact=False, min_clear=0.0)
    finally:
        s.close()


@pytest.mark.parametrize("vocab", [3, 4, 513])
@pytest.mark.parametrize("exact", [True, False])
def test_top_k_bound_beyond_the_float_range(oracle, vocab, exact):
    """A bound whose margin overflows (a huge temperature, logits across the whole f32 range) lists finite logits only:
    what is masked or lies behind the end of a short row stays out of the list."""
    import pagoda_b200
    from pagoda_b200 import synth
    rows = 12
    rng = np.random.default_rng(vocab)
    x = rng.standard_normal((rows, vocab)).astype(np.float32)
    x[6:] = x[6:] / np.abs(x[6:]).max(axis=1, keepdims=True) * np.float32(3.0e38)
    temperature = np.where(np.arange(rows) < 6, np.float32(1e38), np.float32(1.0)).astype(np.float32)
    words = np.full((2, (vocab + 31) // 32), 0xffffffff, np.uint32)
    words[1] &= np.uint32(0xaaaaaaab)
    w = synth.Workload("range", x, temperature, np.resize(np.uint32([1, 2]), rows), np.resize(np.float32([1.0, 0.9]), rows),
                       np.zeros(rows, np.float32), np.zeros(rows, np.float32), np.ones(rows, np.float32), None, None,
                       synth.uniform_f32(9, rows), mask_words=words, state_flags=np.zeros(2, np.uint32),
                       mask_state=np.resize(np.int32([0, 1]), rows))
    s = pagoda_b200.Sampler(device=0, max_rows=rows, max_vocab=vocab, max_history=1)
    try:
        s.set_exact(exact)
        assert_same(*run_both(s, oracle, w), w, exact=exact)
    finally:
        s.close()


def test_a_barrier_that_gives_up_is_reported(monkeypatch):
    """With no polls allowed every wait of the grid barrier runs out: each row that the wide kernel had to do gets a status
    of its own, the counted rows come back as an error code once, and other rows and later calls are not affected."""
    import torch
    import pagoda_b200
    rows, vocab = 6, 65536
    x = torch.randn(rows, vocab, generator=torch.Generator().manual_seed(1))
    kw = dict(temperature=np.float32([0.7, 0.0, 0.7, 0.0, 0.7, 0.7]), top_k=np.zeros(rows, np.uint32),
              top_p=np.full(rows, 0.9, np.float32), uniform=np.full(rows, 0.5, np.float32))
    good = pagoda_b200.Sampler(device=0, max_rows=rows, max_vocab=vocab, max_history=1)
    monkeypatch.setenv("PGS_GRID_POLLS", "0")
    s = pagoda_b200.Sampler(device=0, max_rows=rows, max_vocab=vocab, max_history=1)
    try:
        want = good.sample_batch(x.numpy(), diagnostics=True, **kw)
        assert (want.status == 0).all()
        open_rows = kw["temperature"] > 0
        for _ in range(2):
            got = s.sample_batch(x.numpy(), diagnostics=True, **kw)   # the work list: rows without top-k
            assert got.status.tolist() == np.where(open_rows, 5, 0).tolist()
            assert (got.token[open_rows] == 0).all() and not got.drew.any()
            assert (got.token[~open_rows] == want.token[~open_rows]).all()
            with pytest.raises(pagoda_b200.SamplerError, match="4 rows gave up"):
                s.tp_exchange_status()
            s.tp_exchange_status()                                    # reported once
        s.set_exact(True)
        assert (s.sample_batch(x.numpy(), **kw).status == 5).all()
        ids = torch.zeros(rows, dtype=torch.int32).cuda()
        g, _, status = s.log_softmax(x.cuda(), ids=ids, stream_ptr=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert (status.cpu().numpy() == 5).all() and torch.isnan(g).all()
        with pytest.raises(pagoda_b200.SamplerError, match="12 rows gave up"):
            s.tp_exchange_status()
        good.tp_exchange_status()
    finally:
        s.close()
        good.close()


@pytest.mark.parametrize("route", ["1", "2"])   # the grid on every row; one CTA per row
@pytest.mark.parametrize("rows, vocab, top_k, history", [
    (1, 511, 0, 0), (70, 512, 40, 64), (65, 513, 0, 2048), (5, 1025, 1025, 2049), (3, 33025, 0, 300), (200, 1003, 7, 16)])
def test_both_routes(oracle, monkeypatch, route, rows, vocab, top_k, history):
    """Short rows and many rows are done by one CTA per row, others by the whole grid: either way, at the edges of both."""
    import torch
    import pagoda_b200
    from pagoda_b200 import synth
    x = synth.normal_f32(17 + vocab, rows * vocab, 2.0).reshape(rows, vocab)
    x[:, vocab // 2] = x[:, 0]
    x[-1, 0] = np.nan if rows > 1 else 0.0
    w = synth.Workload(
        "routes", x, np.resize(np.float32([0.7, 0.0, 5.0]), rows), np.full(rows, top_k, np.uint32),
        np.resize(np.float32([0.95, 1.0, 0.3]), rows), np.full(rows, 0.2, np.float32), np.full(rows, 0.1, np.float32),
        np.full(rows, 1.1, np.float32), np.arange(rows + 1, dtype=np.uint32) * history if history else None,
        np.random.default_rng(vocab).integers(0, vocab, rows * history).astype(np.uint32) if history else None,
        synth.uniform_f32(3, rows))
    monkeypatch.setenv("PGS_WIDE_ROUTE", route)
    s = pagoda_b200.Sampler(device=0, max_rows=rows, max_vocab=vocab, max_history=max(history, 1))
    try:
        s.set_exact(True)
        assert_same(*run_both(s, oracle, w), w)
        s.set_exact(False)   # unaligned rows, and the work list
        assert_same(*run_both(s, oracle, w), w, exact=False)
        clean = np.nan_to_num(x)
        ids = np.arange(rows, dtype=np.int32) * (vocab - 1) // max(rows - 1, 1)
        g, full, status = s.log_softmax(torch.from_numpy(clean).cuda(), ids=torch.from_numpy(ids).cuda(), full=True,
                                        stream_ptr=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert (status.cpu().numpy() == 0).all()
        check_scores(oracle, clean, ids, g, full)
    finally:
        s.close()


@pytest.mark.parametrize("route", ["1", "3"])   # the grid, and one CTA per row
@pytest.mark.parametrize("top_k", [0, 3000])
@pytest.mark.parametrize("vocab", [16384, 70001])
def test_open_rows_with_any_top_p(oracle, monkeypatch, route, top_k, vocab):
    """Top-p from below zero (the first entry) to just below one (all but the last few), over the whole vocabulary."""
    import pagoda_b200
    from pagoda_b200 import synth
    monkeypatch.setenv("PGS_WIDE_ROUTE", route)
    top_p = np.float32([0.0, -1.0, -0.0, -1e30, 1e-30, 1e-6, 0.5, 0.994, 0.998, 0.9985, 0.999, 0.9999, 0.999999])
    rows = 2 * len(top_p)
    x = synth.normal_f32(23 + vocab, rows * vocab, 2.0).reshape(rows, vocab)
    x[:, vocab // 2] = x[:, 3] = x.max(axis=1) + np.float32(0.5)   # a tie at the first entry
    w = synth.Workload("top-p", x, np.resize(np.float32([1.0, 0.7, 3.0]), rows), np.full(rows, top_k, np.uint32), np.resize(top_p, rows),
                       np.zeros(rows, np.float32), np.zeros(rows, np.float32), np.ones(rows, np.float32), None, None, synth.uniform_f32(5, rows))
    s = pagoda_b200.Sampler(device=0, max_rows=rows, max_vocab=vocab, max_history=1)
    try:
        s.set_exact(True)
        assert_same(*run_both(s, oracle, w), w)
    finally:
        s.close()


def _us(sampler, x, temperature, top_p):
    """A step's time (the best of several) over open rows with one top-p."""
    import torch
    rows = x.shape[0]
    full = lambda v, dt=torch.float32: torch.full((rows,), v, dtype=dt, device=x.device)  # noqa: E731
    desc = sampler.make_device_desc(x, token=full(0, torch.int32), status=full(0, torch.int32), temperature=full(temperature),
                                    top_k=full(0, torch.int32), top_p=full(top_p), uniform=full(0.5))
    stream = torch.cuda.current_stream().cuda_stream
    best = float("inf")
    for _ in range(6):
        begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        begin.record()
        sampler.launch_device(desc, stream)
        end.record()
        end.synchronize()
        best = min(best, begin.elapsed_time(end) * 1e3)
    return best


@pytest.mark.parametrize("top_p, most", [(0.0, 4.0), (-1.0, 4.0), (0.998, 8.0), (0.9995, 8.0)])
def test_open_rows_with_unusual_top_p_stay_in_the_wide_kernel(top_p, most):
    """They need not much more than rows with a usual top-p (one CTA that sorts the whole row takes 25 times as long)."""
    import torch
    import pagoda_b200
    rows, vocab = 2, 131072
    x = 2.0 * torch.randn(rows, vocab, generator=torch.Generator(device="cuda").manual_seed(2), device="cuda")
    s = pagoda_b200.Sampler(device=0, max_rows=rows, max_vocab=vocab, max_history=1)
    try:
        usual = _us(s, x, 1.0, 0.5)
        assert _us(s, x, 1.0, top_p) < most * usual
    finally:
        s.close()


def _row_below_its_estimate(vocab):
    """Logits of a row whose running probabilities fall behind their plain sum: four large ones, then values a little less than
    half an ulp (of a running value below 1/2) above a whole number of ulps, which every addition rounds down.  Where the plain sum
    passes 1/2 by more than the margin of the estimate the running value is still below it."""
    rng, ulp = np.random.default_rng(0), 2.0 ** -25
    parts, mass, m = [np.full(4, 0.065)], 0.26, 44
    while mass < 0.5036:
        near = mass > 0.4965   # few to a bucket here
        n = 1200 if near else min(30000, int((0.497 - mass) / (m + 0.4) / ulp) + 1)
        parts.append((m + rng.uniform(0.02 if near else 0.3, 0.44, n)) * ulp)
        mass += parts[-1].sum()
        m -= 1
    n = vocab - sum(len(q) for q in parts)
    parts.append(np.linspace(m + 0.9, 2.0 * (1.0 - mass) / n / ulp - m - 0.9, n) * ulp)
    p = np.sort(np.concatenate(parts))[::-1]
    where = rng.permutation(vocab)
    x, scale = np.zeros(vocab, np.float32), 1.0
    for _ in range(4):   # (the sum that they are divided by is a fold as well)
        e = np.minimum(p / p[0] * scale, 1.0)
        e[:4] = 1.0
        x[where] = np.log(e)
        scale = np.add.accumulate(np.exp(x.astype(np.float64)).astype(np.float32), dtype=np.float32)[-1] * p[0]
    return x


def test_top_p_where_the_running_value_is_not_as_estimated(oracle, monkeypatch):
    """The fold towards top-p goes on behind a run of buckets that turns out to be in another binade: bit-exact, and in a fraction
    of the time of one CTA that sorts the whole row."""
    import torch
    import pagoda_b200
    from pagoda_b200 import synth
    vocab = 1 << 20
    x = np.stack([_row_below_its_estimate(vocab)])
    w = synth.Workload("estimate", x, np.float32([1.0]), np.uint32([0]), np.float32([0.9]), np.zeros(1, np.float32), np.zeros(1, np.float32),
                       np.ones(1, np.float32), None, None, synth.uniform_f32(5, 1))
    us = {}
    for route in ("1", "2", "3"):
        monkeypatch.setenv("PGS_WIDE_ROUTE", route)
        s = pagoda_b200.Sampler(device=0, max_rows=1, max_vocab=vocab, max_history=1)
        try:
            s.set_exact(True)
            assert_same(*run_both(s, oracle, w), w)
            us[route] = _us(s, torch.from_numpy(x).cuda(), 1.0, 0.9)
        finally:
            s.close()
    assert us["1"] < 0.5 * us["2"] and us["3"] < 0.5 * us["2"], us
