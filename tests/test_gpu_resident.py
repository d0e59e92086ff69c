"""The resident row kernel against the checker where its ways to a cut part: buckets with more
members than a list holds (rows of few values), all candidates in one slice (rows sorted by id),
cuts by a large top_k, min_p between two cuts, vocabularies at the edges of a slice."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from tests.test_gpu_parity import compare_case, general_sampler, sampler  # noqa: E402,F401


def _rows(kind, rng, batch, vocab):
    x = (rng.standard_normal((batch, vocab)) * 2.5).astype(np.float32)
    if kind == "few values":
        return (np.round(x) * 0.5).astype(np.float32)
    if kind == "sorted by id":
        return -np.sort(-x, axis=1)
    if kind == "constant":
        return np.full((batch, vocab), 1.25, np.float32)
    if kind == "far apart":
        return (x * 40).astype(np.float32)
    return x


@pytest.mark.parametrize("vocab", [7, 4_095, 33_001, 65_536])
@pytest.mark.parametrize("kind", ["normal", "few values", "sorted by id", "constant", "far apart"])
def test_every_way_to_a_cut_matches_the_checker(sampler, general_sampler, kind, vocab):  # noqa: F811
    from hydraserve_b200.engine.sampling import SamplingParams
    from hydraserve_b200.workloads import Workload

    rng = np.random.default_rng(vocab)
    params = [SamplingParams(temperature=1.0, top_p=0.9, seed=1, logprobs=20),
              SamplingParams(temperature=0.7, top_k=300, top_p=0.95, seed=2, logprobs=5, presence_penalty=0.4),
              SamplingParams(temperature=1.3, min_p=0.02, top_p=0.8, seed=3, repetition_penalty=1.2),
              SamplingParams(temperature=1.0, top_k=40, top_p=0.9, seed=4, frequency_penalty=0.3, logprobs=20),
              SamplingParams(temperature=0.0, logprobs=20, presence_penalty=0.6)]
    hist = [rng.integers(0, vocab, 600).astype(np.int32) for _ in params]
    w = Workload(kind, _rows(kind, rng, len(params), vocab), "f32", hist, params, [5] * len(params))
    compare_case(sampler, w).assert_ok(max_sensitive_fraction=0.6)
    compare_case(general_sampler, w).assert_ok(max_sensitive_fraction=0.6)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("heavy", [1, 2_000])
def test_the_lowest_id_wins_a_tie_with_tokens_held_three_times(built_library, dtype, heavy):
    """Penalised arg max: `heavy` tokens held three times and one other all score exactly 5; the
    lowest id among them is a heavy one (with 2,000, a thread meets several of them, in any order)."""
    from hydraserve_b200.engine import SamplingParams, sample_logits

    vocab = 32_768
    ids = 5 + np.arange(heavy)
    logits = torch.full((2, vocab), -1.0)
    logits[:, ids] = 8.0
    logits[:, 2_048] = 5.0
    history = np.repeat(ids[::-1], 3).tolist()
    params = [SamplingParams(frequency_penalty=1.0), SamplingParams(frequency_penalty=1.0, logprobs=3)]
    got = sample_logits(logits.to(dtype).cuda(), [history] * 2, params, steps=[0, 0])
    assert [s.token_id for s in got] == [5, 5]
