"""fp32 batches of more rows than clusters hold side by side (rows with a small top_k are streamed, the
others resident) against the checker: rows off the 16-byte boundary, too few tokens for a first
bound, ties that overflow a list, every row of one kind."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from tests.test_gpu_parity import compare_case  # noqa: E402


@pytest.fixture(scope="module")
def sampler(built_library):
    from hydraserve_b200.engine import _device

    s = _device.DeviceSampler("cuda:0", vocab_max=33_003, batch_max=600, resident_slots=1)
    yield s
    s.close()


@pytest.mark.parametrize("kind,vocab,batch", [("mixed", 33_001, 75), ("mixed", 32_768, 75), ("small top_k", 33_003, 76),
                                              ("others", 32_770, 75), ("ties", 33_001, 75), ("mixed", 4_099, 600)])
def test_streamed_and_resident_rows_match_the_checker(sampler, kind, vocab, batch):
    from hydraserve_b200.engine.sampling import SamplingParams
    from hydraserve_b200.workloads import Workload

    rng = np.random.default_rng(vocab + batch)
    x = (rng.standard_normal((batch, vocab)) * 2.5).astype(np.float32)
    if kind == "ties":
        x = np.minimum(np.round(x), 1).astype(np.float32)
    small = [SamplingParams(temperature=0.8, top_k=1, seed=1),
             SamplingParams(temperature=0.7, top_k=50, top_p=0.9, seed=2, repetition_penalty=1.1),
             SamplingParams(temperature=1.2, top_k=256, min_p=0.01, seed=3, logprobs=20, presence_penalty=0.4),
             SamplingParams(temperature=1.0, top_k=20, seed=4, frequency_penalty=0.3, logprobs=5)]
    others = [SamplingParams(temperature=0.0, logprobs=3, presence_penalty=0.6),
              SamplingParams(temperature=1.0, top_p=0.9, seed=5),
              SamplingParams(temperature=1.0, top_k=257, seed=6)]
    cycle = {"small top_k": small, "others": others}.get(kind, small + others)
    params = [cycle[i % len(cycle)] for i in range(batch)]
    hist = [rng.integers(0, vocab if i % 2 else 40, 300).astype(np.int32) for i in range(batch)]
    w = Workload(kind, x, "f32", hist, params, [i % 9 for i in range(batch)])
    compare_case(sampler, w).assert_ok(max_sensitive_fraction=0.6)
