"""Rows with a small top_k whose candidates do not fit a list on the way (scores that rise with the
id, penalties that raise scores): which token a seed names is a matter of the row alone, whatever
the batch around it and however many CTAs share the row."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from hydraserve_b200.engine import SamplingParams, sample_logits, sample_logits_packed  # noqa: E402


@pytest.fixture(autouse=True)
def _lib(built_library):
    return built_library


def _row(kind, vocab, dtype):
    """(logits of the row, its history, its parameters beside the seed)"""
    x = torch.randn(vocab, generator=torch.Generator().manual_seed(vocab)) * 3
    if kind == "rising":
        return x.sort().values.to(dtype), [], {}
    if kind == "rising at the end":  # (only the last CTA of a split row has a crowded list)
        x[-vocab // 9:] = x[-vocab // 9:].sort().values + 4
        return x.to(dtype), [], {}
    if kind == "ties":  # more at the k-th score than a list holds
        return x.clamp(max=0.5).to(dtype), [], {}
    # a token of the history would need a score this low to count
    return x.to(dtype), [1, 2, 3, 3, 3], dict(presence_penalty=-2.0, repetition_penalty=0.5, frequency_penalty=-2.0)


@pytest.mark.parametrize("kind", ["rising", "rising at the end", "ties", "raised scores"])
@pytest.mark.parametrize("vocab", [32_768, 65_541, 151_936])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_a_seeded_row_draws_the_same_token_in_every_batch(dtype, vocab, kind):
    row, history, more = _row(kind, vocab, dtype)
    params = [SamplingParams(temperature=1.0, top_k=50, seed=100 + i, **more) for i in range(8)]
    tokens = {}
    for batch in (1, 8, 80, 256):
        logits = row.cuda().expand(batch, vocab).contiguous()
        rows = [sample_logits(logits, [history] * batch, [params[(i + t) % 8] for i in range(batch)], steps=[3] * batch)
                for t in range(8 if batch < 8 else 1)]
        for t, samples in enumerate(rows):
            for i, s in enumerate(samples):
                tokens.setdefault((i + t) % 8, set()).add(s.token_id)
    assert all(len(t) == 1 for t in tokens.values()), tokens


@pytest.mark.parametrize("kind", ["rising", "ties", "raised scores"])
@pytest.mark.parametrize("batch", [1, 80])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_counts_and_log_probabilities_of_a_crowded_row(dtype, batch, kind):
    """The filters and the log-probabilities against torch in 64 bits."""
    vocab, k = 65_541, 50
    row, history, more = _row(kind, vocab, dtype)
    score = row.double().clone()
    for t in set(history):
        n = history.count(t)
        v = score[t] * (0.5 if score[t] < 0 else 2.0) + 2.0 + 2.0 * n
        score[t] = v.float().double()
    kth = score.topk(k).values[-1]
    kept = torch.nonzero(score >= kth).flatten()
    order = sorted(kept.tolist(), key=lambda i: (-float(score[i]), i))
    logp = torch.log_softmax(score[kept], 0)
    by_id = dict(zip(kept.tolist(), logp.tolist()))
    logits = row.cuda().expand(batch, vocab).contiguous()
    params = [SamplingParams(temperature=1.0, top_k=k, seed=7 + i, logprobs=20, **more) for i in range(batch)]
    got = sample_logits_packed(logits, [history] * batch, params, steps=[1] * batch)
    assert (got.records["n_kept"] == len(kept)).all() and (got.records["status"] == 0).all()
    for s in got:
        assert s.token_id in by_id
        # (sums of 2**-40 units behind a 32-bit logarithm: a few ulp of values up to 16)
        assert abs(s.logprob - by_id[s.token_id]) < 1e-5
        assert [t for t, _ in s.top_logprobs] == order[:20]
        np.testing.assert_allclose([v for _, v in s.top_logprobs], [by_id[t] for t in order[:20]], rtol=0, atol=1e-5)


@pytest.mark.parametrize("slope", [1.0, 4.0, 16.0])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_lists_that_are_looked_at_after_every_batch_of_loads(dtype, slope):
    """Rows that drift upwards list hundreds of tokens per batch of loads, so the stream looks at
    its list after every batch, one barrier behind the other; the candidates against torch."""
    from hydraserve_b200.engine.sharded import sample_logits_sharded

    vocab, batch, k = 248_320, 80, 56
    x = torch.randn((batch, vocab), generator=torch.Generator().manual_seed(int(slope))) + torch.linspace(0, slope, vocab)
    logits = x.to(dtype).cuda()
    kth = logits.topk(k, dim=1).values[:, -1:]
    kept = (logits >= kth).sum(1).tolist()
    params = [SamplingParams(temperature=1.0, top_k=k, seed=i) for i in range(batch)]
    first = sample_logits_packed(logits, [[]] * batch, params, steps=[0] * batch)
    assert first.records["n_kept"].tolist() == kept and not first.records["status"].any()
    tokens = torch.from_numpy(first.token_ids.astype(np.int64)).cuda()[:, None]
    assert (logits.gather(1, tokens) >= kth).all()
    for _ in range(20):
        again = sample_logits_packed(logits, [[]] * batch, params, steps=[0] * batch)
        assert again.token_ids.tolist() == first.token_ids.tolist()
    if dtype == torch.bfloat16 and max(kept) <= 64:  # (the candidates of a slice that one record holds)
        sharded = sample_logits_sharded(logits, [[]] * batch, params, steps=[0] * batch, vocab_offset=0, vocab_total=vocab)
        assert [s.token_id for s in sharded] == first.token_ids.tolist()


def test_what_a_record_does_not_use_is_zero():
    """Rows that went through a kernel a second time, and rows with fewer candidates than
    log-probabilities: a packed result carries nothing of other rows or earlier steps."""
    vocab, batch = 151_936, 80
    row, _, _ = _row("rising", vocab, torch.float32)
    logits = row.cuda().expand(batch, vocab).contiguous()
    full = [SamplingParams(temperature=1.0, top_k=50, seed=i, logprobs=20) for i in range(batch)]
    none = [SamplingParams(temperature=1.0, top_k=50, seed=i) for i in range(batch)]
    few = [SamplingParams(temperature=1.0, top_k=3, seed=i, logprobs=20) for i in range(batch)]
    normal = torch.randn(batch, vocab, generator=torch.Generator().manual_seed(3)).cuda()
    for x in (logits, normal):
        for params, used in ((full, 20), (none, 0), (few, 3)):
            records = sample_logits_packed(x, [[]] * batch, params, steps=[0] * batch).records
            assert (records["n_top"] == used).all()
            assert not records["top_ids"][:, used:].any() and not records["top_logprobs"][:, used:].any()
