"""The streaming kernel against the oracle where its branches change: candidate lists around the lengths of the sort,
histories that crowd one 512-logit region or fill the table, masks that end inside a word, a bf16 row of odd groups."""
import numpy as np
import pytest

from .util import assert_close, run_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vocab, top_k, history, crowd, masked, bf16", [
    (8200, 255, 40, 512, False, False), (8192, 257, 2048, 8192, True, False), (40016, 511, 300, 300, True, True),
    (32776, 513, 700, 32776, False, True), (151936, 1024, 1, 1, True, False), (262144, 1000, 2047, 1024, False, False),
    (262152, 64, 8, 64, True, True)])
def test_stream_edges(oracle, vocab, top_k, history, crowd, masked, bf16):
    import pagoda_b200
    from pagoda_b200 import synth
    rows = 6
    rng = np.random.default_rng(vocab + top_k)
    x = synth.normal_f32(11 + vocab, rows * vocab, 2.0).reshape(rows, vocab)
    x[:, rng.integers(0, vocab, 40)] += 6.0
    kw = {}
    if masked:
        words = rng.integers(0, 1 << 32, (3, (vocab + 31) // 32), dtype=np.uint64).astype(np.uint32)
        kw = dict(mask_words=words, state_flags=np.array([0, 1, 0], np.uint32),
                  mask_state=np.array([0, 1, 2, -1, 1, 0], np.int32), eos_token_id=vocab - 1)
    w = synth.Workload(
        "edges", (x.view(np.uint32) >> 16).astype(np.uint16) if bf16 else x, np.resize(np.float32([0.7, 1.3, 0.0]), rows),
        np.full(rows, top_k, np.uint32), np.resize(np.float32([1.0, 0.9]), rows), np.full(rows, 0.2, np.float32),
        np.full(rows, 0.1, np.float32), np.full(rows, 1.1, np.float32), np.arange(rows + 1, dtype=np.uint32) * history,
        rng.integers(0, crowd, rows * history).astype(np.uint32), synth.uniform_f32(5, rows), **kw)
    s = pagoda_b200.Sampler(device=0, max_rows=rows, max_vocab=vocab, max_history=history)
    try:
        assert_close(*run_both(s, oracle, w), "edges")
    finally:
        s.close()


def _batch(rows, vocab, top_k, history, crowd, masked, bf16):
    from pagoda_b200 import synth
    rng = np.random.default_rng(vocab + top_k + rows)
    x = synth.normal_f32(13 + vocab, rows * vocab, 2.0).reshape(rows, vocab)
    x[:, rng.integers(0, vocab, 40)] += 6.0
    x[:, vocab - 1] = x[:, 0]
    kw = {}
    if masked:
        words = rng.integers(0, 1 << 32, (3, (vocab + 31) // 32), dtype=np.uint64).astype(np.uint32)
        kw = dict(mask_words=words, state_flags=np.array([0, 1, 0], np.uint32),
                  mask_state=np.resize(np.int32([0, 1, 2, -1, 1, 0]), rows), eos_token_id=vocab - 1)
    return synth.Workload(
        "edges", (x.view(np.uint32) >> 16).astype(np.uint16) if bf16 else x, np.resize(np.float32([0.7, 1.3, 0.0]), rows),
        np.full(rows, top_k, np.uint32), np.resize(np.float32([1.0, 0.9]), rows), np.full(rows, 0.2, np.float32),
        np.full(rows, 0.1, np.float32), np.full(rows, 1.1, np.float32),
        np.arange(rows + 1, dtype=np.uint32) * history if history else None,
        rng.integers(0, crowd, rows * history).astype(np.uint32) if history else None, synth.uniform_f32(5, rows), **kw)


# Rows on a cluster of CTAs each, and on one CTA each; 330 rows: more than are resident, so that a CTA takes a second row and
# its tables and bits are used again.
@pytest.mark.parametrize("cluster", ["1", "0"])
@pytest.mark.parametrize("rows, vocab, top_k, history, crowd, masked, bf16", [
    (330, 8200, 255, 40, 512, False, False), (330, 4096, 40, 2048, 4096, True, True), (330, 1000, 20, 512, 1000, False, False),
    (24, 8192, 257, 2048, 8192, True, False), (24, 40016, 511, 300, 300, True, True), (16, 50256, 1024, 100, 50256, False, False),
    (24, 32776, 513, 700, 32776, False, True), (12, 151936, 1024, 1, 1, True, False)])
def test_stream_edges_on_one_cta_and_on_clusters(oracle, monkeypatch, cluster, rows, vocab, top_k, history, crowd, masked, bf16):
    import pagoda_b200
    monkeypatch.setenv("PGS_CLUSTER", cluster)
    w = _batch(rows, vocab, top_k, history, crowd, masked, bf16)
    s = pagoda_b200.Sampler(device=0, max_rows=rows, max_vocab=vocab, max_history=history)
    try:
        assert_close(*run_both(s, oracle, w), "edges")
    finally:
        s.close()


# bf16 rows whose masked logits are the largest by far: one CTA per row adds -inf to them, rows of a cluster and longer ones select.
@pytest.mark.parametrize("cluster", ["1", "0"])
@pytest.mark.parametrize("vocab, greedy", [(1000, False), (8200, False), (40016, True), (262152, False)])
def test_masked_logits_that_are_the_largest(oracle, monkeypatch, cluster, vocab, greedy):
    import pagoda_b200
    monkeypatch.setenv("PGS_CLUSTER", cluster)
    rows = 9
    w = _batch(rows, vocab, 40, 30, vocab, True, True)
    x = w.logits_f32().copy()
    for r, state in enumerate(w.mask_state):
        if state >= 0:
            allowed = np.unpackbits(w.mask_words[state].view(np.uint8), bitorder="little")[:vocab].astype(bool)
            x[r, ~allowed] += 1000.0 * (1 + r)
    w.logits[...] = (x.astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
    if greedy:
        w.temperature[...] = 0.0
    s = pagoda_b200.Sampler(device=0, max_rows=rows, max_vocab=vocab, max_history=30)
    try:
        assert_close(*run_both(s, oracle, w), "masked", min_clear=0.0)
    finally:
        s.close()


# Long candidate lists are folded in runs of sixteen, short ones by one lane.
@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("rows, vocab, top_k", [(5, 4096, 160), (5, 40000, 161), (9, 151936, 500), (300, 8192, 700)])
def test_top_p_of_zero_keeps_the_first_entry(oracle, exact, rows, vocab, top_k):
    """top_p <= 0 is reached behind the first entry (sampler.rs:136-144), whatever was in shared memory before (the raw logits of
    the history, which are negative)."""
    import pagoda_b200
    from pagoda_b200 import synth
    x = synth.normal_f32(19 + vocab, rows * vocab, 2.0).reshape(rows, vocab) - np.float32(30.0)
    x[:, vocab // 2] = x[:, 3]
    w = synth.Workload(
        "zero", x, np.resize(np.float32([0.7, 1.0, 4.0]), rows), np.full(rows, top_k, np.uint32),
        np.resize(np.float32([0.0, -1.0, -0.0, -1e30, 1e-30]), rows), np.full(rows, 0.2, np.float32), np.full(rows, 0.1, np.float32),
        np.ones(rows, np.float32), np.arange(rows + 1, dtype=np.uint32) * 2048,
        np.stack([np.random.default_rng(r).permutation(vocab)[:2048] for r in range(rows)]).astype(np.uint32).ravel(), synth.uniform_f32(5, rows))
    s = pagoda_b200.Sampler(device=0, max_rows=rows, max_vocab=vocab, max_history=2048)
    try:
        s.set_exact(exact)
        for _ in range(2):
            got, want = run_both(s, oracle, w)
            assert (want["n_kept"] == 1).all()
            for name in ("status", "token", "n_kept", "argmax"):
                np.testing.assert_array_equal(getattr(got, name), want[name], err_msg=name)
            np.testing.assert_allclose(got.total, want["total"], rtol=1e-5)
    finally:
        s.close()


# Rows whose bits do not fit in shared memory, from the first length on to the longest.
@pytest.mark.parametrize("cluster", ["1", "0"])
@pytest.mark.parametrize("vocab, top_k, history, crowd, masked, bf16", [
    (262152, 64, 8, 64, True, True), (262152, 50, 0, 1, False, False), (262148, 1000, 2047, 262148, True, False),
    (300008, 40, 600, 700, False, True), ((1 << 20) - 4, 20, 2048, 1 << 20, False, False), (1 << 20, 50, 100, 1 << 20, True, True)])
def test_stream_long_rows(oracle, monkeypatch, cluster, vocab, top_k, history, crowd, masked, bf16):
    import pagoda_b200
    monkeypatch.setenv("PGS_CLUSTER", cluster)
    rows = 9
    w = _batch(rows, vocab, top_k, history, crowd, masked, bf16)
    s = pagoda_b200.Sampler(device=0, max_rows=rows, max_vocab=vocab, max_history=max(history, 1))
    try:
        assert_close(*run_both(s, oracle, w), "long rows")
    finally:
        s.close()
