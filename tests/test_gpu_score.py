"""`sampler::log_softmax` (sampler.rs:73-87) and the gather of `Engine::score` on the device against
the oracle.  exp and the f32 left-fold sum are exact; ln is the double logarithm rounded to f32, so
the comparison allows 1e-6 (absolute, values are O(10))."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_log_softmax_matches_oracle(oracle):
    import torch
    import pagoda_b200
    from pagoda_b200 import synth
    s = pagoda_b200.Sampler(device=0, max_rows=8, max_vocab=151936, max_history=16)
    st = torch.cuda.current_stream().cuda_stream
    try:
        for rows, vocab, std in ((3, 3, 1.0), (6, 1000, 2.0), (4, 151936, 3.0)):
            x = synth.normal_f32(40 + vocab, rows * vocab, std).reshape(rows, vocab)
            if vocab == 3:
                x[0] = [0.0, 1.0, 2.0]                      # sampler.rs:231-235 log_softmax_sums_to_one
                x[1] = [5.0, 5.0 - 200.0, 5.0 - 300.0]      # sum == 1: the MIN_POSITIVE clamp; ln(0) = -inf
            ids = np.arange(rows, dtype=np.int32) % vocab
            g, full, status = s.log_softmax(torch.from_numpy(x).cuda(), ids=torch.from_numpy(ids).cuda(), full=True,
                                            stream_ptr=st)
            torch.cuda.synchronize()
            full, g = full.cpu().numpy(), g.cpu().numpy()
            assert (status.cpu().numpy() == 0).all()
            for r in range(rows):
                want = oracle.log_softmax(x[r])
                fin = np.isfinite(want)
                np.testing.assert_array_equal(np.isfinite(full[r]), fin)
                np.testing.assert_allclose(full[r][fin], want[fin], rtol=0, atol=1e-6 * max(1.0, np.abs(want[fin]).max()))
                assert g[r] == full[r][ids[r]]
            if vocab == 3:
                assert abs(np.exp(full[0].astype(np.float64)).sum() - 1.0) < 1e-6
        bad = np.zeros((2, 64), np.float32)
        bad[1, 3] = np.nan
        g, _, status = s.log_softmax(torch.from_numpy(bad).cuda(), ids=torch.zeros(2, dtype=torch.int32).cuda(), stream_ptr=st)
        torch.cuda.synchronize()
        assert status.cpu().numpy().tolist() == [0, 1] and np.isnan(g.cpu().numpy()[1])
    finally:
        s.close()


@pytest.mark.parametrize("rows, vocab", [(3, 511), (3, 20001), (64, 50257), (65, 120001), (200, 131072)])
def test_more_rows_than_the_handle_was_made_for(oracle, rows, vocab):
    """Scoring has no row limit: the rows of a call beyond what the workspace holds are taken in turn."""
    import torch
    import pagoda_b200
    from pagoda_b200 import synth
    x = synth.normal_f32(70 + rows, rows * vocab, 3.0).reshape(rows, vocab)
    ids = np.random.default_rng(rows).integers(0, vocab, rows).astype(np.int32)
    s = pagoda_b200.Sampler(device=0, max_rows=2, max_vocab=vocab, max_history=1)
    try:
        g, full, status = s.log_softmax(torch.from_numpy(x).cuda(), ids=torch.from_numpy(ids).cuda(), full=True,
                                        stream_ptr=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        full, g = full.cpu().numpy(), g.cpu().numpy()
        assert (status.cpu().numpy() == 0).all()
        for r in range(rows):
            want = oracle.log_softmax(x[r])
            np.testing.assert_allclose(full[r], want, rtol=0, atol=1e-6 * np.abs(want).max())
            assert g[r] == full[r][ids[r]]
    finally:
        s.close()


def test_scoring_keeps_nothing_of_the_stream_it_ran_on():
    """Scoring on one stream does not wait for the handle's work on another, can be captured whatever ran before, and the
    stream may be gone when the handle is used again; every route gives the same bits."""
    import ctypes
    import torch
    import pagoda_b200
    rows, vocab = 16, 50257
    x = torch.randn(rows, vocab, generator=torch.Generator().manual_seed(5)).cuda() * 3
    ids = torch.arange(rows, dtype=torch.int32).cuda() * 3000
    other, busy = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    s = pagoda_b200.Sampler(device=0, max_rows=rows, max_vocab=vocab, max_history=1)
    token, status = torch.zeros(rows, dtype=torch.int32).cuda(), torch.zeros(rows, dtype=torch.int32).cuda()
    step = s.make_device_desc(x, token=token, status=status)

    def score(stream):
        with torch.cuda.stream(stream):
            g, full, st = s.log_softmax(x, ids=ids, full=True, stream_ptr=stream.cuda_stream)
            return torch.cat([g[:, None], full], 1), st

    try:
        want, st = score(other)
        other.synchronize()
        assert (st == 0).all()
        # captured on a stream that is not the handle's last one
        s.launch_device(step, busy.cuda_stream)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=other):
            captured, _ = score(other)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(captured, want)
        # a step and a scoring call behind a long kernel on one stream, scoring on another
        with torch.cuda.stream(busy):
            torch.cuda._sleep(1 << 30)
        s.launch_device(step, busy.cuda_stream)
        late, _ = score(busy)
        again, _ = score(busy)
        now, _ = score(other)
        other.synchronize()
        assert not busy.query()
        assert torch.equal(now, want)
        busy.synchronize()
        assert torch.equal(late, want) and torch.equal(again, want)
        # a stream that is destroyed afterwards
        rt, raw = torch.cuda.cudart(), ctypes.c_void_p()
        assert rt.cudaStreamCreate(ctypes.addressof(raw)) == 0
        gone, _ = score(torch.cuda.ExternalStream(raw.value))
        torch.cuda.synchronize()
        assert rt.cudaStreamDestroy(raw.value) == 0
        assert torch.equal(gone, want)
        s.launch_device(step, other.cuda_stream)
        last, _ = score(busy)
        torch.cuda.synchronize()
        assert torch.equal(last, want) and torch.equal(token.long(), x.argmax(1))
    finally:
        s.close()


def test_both_kernels_score_alike():
    """Short rows and batches of many rows are scored by one CTA per row, others by the whole grid: the same row gives the
    same bits in batches on either side of the line."""
    import torch
    import pagoda_b200
    st = torch.cuda.current_stream().cuda_stream
    for vocab, many, few in ((16384, 128, 64), (50257, 128, 64), (4096, 64, 1), (20000, 64, 1)):
        x = torch.randn(many, vocab, generator=torch.Generator().manual_seed(vocab)).cuda() * 3
        ids = torch.arange(many, dtype=torch.int32).cuda() * 7
        s = pagoda_b200.Sampler(device=0, max_rows=4, max_vocab=vocab, max_history=1)
        try:
            for full in (False, True):
                a = s.log_softmax(x, ids=ids, full=full, stream_ptr=st)
                b = s.log_softmax(x[:few], ids=ids[:few], full=full, stream_ptr=st)
                torch.cuda.synchronize()
                assert torch.equal(a[0][:few], b[0]) and (a[2] == 0).all()
                if full:
                    assert torch.equal(a[1][:few], b[1])
        finally:
            s.close()
