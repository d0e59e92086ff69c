"""The host-to-host step (hs_step: histories counted by one launch, parameters and single tokens in the
launches themselves) against the step made of its parts (slots_append and hs_sample), at history
lengths around what a thread, a CTA and a cluster take at once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from hydraserve_b200.engine import SamplingParams, release_request, sample_logits  # noqa: E402

VOCAB = 30_000


@pytest.mark.parametrize("batch", [1, 3, 65])
@pytest.mark.parametrize("length", [1, 2, 33, 512, 2_049, 16_385, 40_000])
def test_step_equals_its_parts(built_library, batch, length):
    from hydraserve_b200.engine import _device

    rng = np.random.default_rng(length)
    logits = torch.from_numpy(rng.standard_normal((batch, VOCAB)).astype(np.float32)).cuda().bfloat16()
    params = [SamplingParams(temperature=[0.0, 1.0][i % 2], top_p=0.9, seed=i, logprobs=20, repetition_penalty=1.1,
                             presence_penalty=0.5, frequency_penalty=0.3) for i in range(batch)]
    # (some ids very often, some outside the vocabulary)
    histories = [np.where(rng.random(length) < 0.3, rng.integers(0, 40, length),
                          rng.integers(-3, VOCAB + 3, length)).tolist() for _ in range(batch)]
    ids = [("step", i) for i in range(batch)]
    parts = _device.DeviceSampler("cuda:0", vocab_max=VOCAB, batch_max=batch, resident_slots=batch, hist_cap=VOCAB)
    try:
        for grow in (0, 1, 3, 1, 2_000):
            for h in histories:
                h.extend(int(t) for t in rng.integers(0, 60, grow))
            records, _ = parts.sample(logits, histories, params, [grow] * batch, None)
            want = _device.records_to_samples(records, params, VOCAB)
            assert sample_logits(logits, histories, params, steps=[grow] * batch, request_ids=ids) == want
            assert sample_logits(logits, histories, params, steps=[grow] * batch) == want
    finally:
        parts.close()
        for i in ids:
            release_request(i)
