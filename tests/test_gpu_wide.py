"""The wide kernel (exact mode, unaligned rows, wide-open rows, scoring) against the oracle, at the edges of its
512-logit regions, of its row chunk, of the candidate list that one CTA finishes and of the history it takes."""
import numpy as np
import pytest

from .util import assert_same, run_both

pytestmark = pytest.mark.gpu


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
        for r in range(min(rows, 3)):
            np.testing.assert_allclose(full[r].cpu().numpy(), oracle.log_softmax(x[r]), rtol=0, atol=2e-5)
            assert g[r] == full[r][int(ids[r])]
    finally:
        s.close()
