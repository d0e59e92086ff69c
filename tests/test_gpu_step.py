"""The host-to-host step (hs_step: histories counted by one launch, parameters and single tokens in the
launches themselves) against the step made of its parts (slots_append and hs_sample), at history
lengths around what a thread, a CTA and a cluster take at once."""
import ctypes as C

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


class _Desc(C.Structure):
    _fields_ = [(n, C.c_size_t) for n in ("bytes", "resets_at", "slots_at", "offsets_at", "tokens_at")] + \
               [(n, C.c_int32) for n in ("n_resets", "n_appends", "max_tokens", "repeats")]


def test_a_wait_is_for_the_step_before_it(built_library):
    """hs_step and hs_step_greedy may be followed by the caller's own wait instead of hs_step_wait:
    a later step's hs_step_wait then waits for that step's results, all of them and no others."""
    from hydraserve_b200 import _lib
    from hydraserve_b200.engine import _device

    batch = 8
    s = _device.DeviceSampler("cuda:0", vocab_max=VOCAB, batch_max=batch, resident_slots=1)
    rec = _device.pack_params([SamplingParams(temperature=1.0, top_k=1, seed=i) for i in range(batch)], [0] * batch)
    stream = s._stream()
    logits, records = None, None  # (of the step; where the sampler's records stand)

    def rows(seed):  # and where each has its maximum
        gen = torch.Generator().manual_seed(seed)
        x, best = torch.randn(batch, VOCAB, generator=gen), torch.randint(0, VOCAB, (batch,), generator=gen)
        x[range(batch), best] = 9.0
        return x.cuda().bfloat16(), best.tolist()

    def sample():
        nonlocal records
        if records:  # (nothing of an earlier step is left there)
            C.memset(records, 0x55, batch * 208)
        block, out = C.c_void_p(), C.c_void_p()
        assert s.lib.hs_step_block(s.handle, rec.nbytes, C.byref(block)) == 0
        C.memmove(block.value, rec.ctypes.data, rec.nbytes)
        d = _Desc(rec.nbytes, rec.nbytes, rec.nbytes, rec.nbytes, rec.nbytes, 0, 0, 0, 0)
        assert s.lib.hs_step(s.handle, logits.data_ptr(), 1, VOCAB, batch, VOCAB, C.byref(d), C.byref(out), stream) == 0
        records = out.value
        return lambda: np.frombuffer((C.c_char * (batch * 208)).from_address(records), dtype=_lib.ROW_OUT)

    def greedy():
        out = C.c_void_p()
        assert s.lib.hs_step_greedy(s.handle, logits.data_ptr(), 1, VOCAB, batch, VOCAB, C.byref(out), stream) == 0
        return lambda: np.frombuffer((C.c_int32 * batch).from_address(out.value), dtype=np.int32)

    try:
        for step, first in enumerate((greedy, sample, greedy, sample, greedy)):
            logits, _ = rows(2 * step)
            first()
            torch.cuda.synchronize()  # (the caller's own wait)
            logits, best = rows(2 * step + 1)
            torch.cuda._sleep(2_000_000)  # a millisecond: the results cannot be there by themselves
            second = sample if first is greedy else greedy
            read = second()
            assert s.lib.hs_step_wait(s.handle, stream) == 0
            got = read().copy()
            if second is sample:
                assert not got["status"].any() and got["token"].tolist() == best
            else:
                assert got.tolist() == best
            torch.cuda.synchronize()
    finally:
        s.close()


@pytest.mark.parametrize("repeats", [0, 1, -1])
def test_records_of_a_step_its_caller_waits_for(built_library, repeats):
    """hs_step without hs_step_wait: at the stream's end the records stand where *out points, whatever
    number says that a slot is listed twice."""
    from hydraserve_b200 import _lib
    from hydraserve_b200.engine import _device

    vocab, batch = 5_000, 6
    params = [SamplingParams(temperature=1.0, top_k=(0, 40)[i % 2], seed=i, logprobs=(None, 5, None)[i % 3]) for i in range(batch)]
    s = _device.DeviceSampler("cuda:0", vocab_max=vocab, batch_max=batch, resident_slots=1)
    out = C.c_void_p()
    try:
        for step in range(3):
            logits = torch.randn(batch, vocab, generator=torch.Generator().manual_seed(step)).cuda().bfloat16()
            rec = _device.pack_params(params, [step] * batch, [-1] * batch)
            want, _ = s.run(logits, rec)
            if out.value:
                C.memset(out.value, 0x55, batch * _lib.ROW_OUT.itemsize)  # (no record of an earlier step)
            block = C.c_void_p()
            assert s.lib.hs_step_block(s.handle, rec.nbytes, C.byref(block)) == 0
            C.memmove(block.value, rec.ctypes.data, rec.nbytes)
            d = _Desc(rec.nbytes, rec.nbytes, rec.nbytes, rec.nbytes, rec.nbytes, 0, 0, 0, repeats)
            assert s.lib.hs_step(s.handle, logits.data_ptr(), 1, vocab, batch, vocab, C.byref(d), C.byref(out), s._stream()) == 0
            torch.cuda.synchronize()
            got = np.frombuffer((C.c_char * (batch * _lib.ROW_OUT.itemsize)).from_address(out.value), dtype=_lib.ROW_OUT)
            for i in range(batch):
                for name in _lib.ROW_OUT.names:
                    if params[i].logprobs is not None or not name.startswith("top_"):
                        np.testing.assert_array_equal(got[i][name], want[i][name], err_msg=f"{name} of row {i}")
    finally:
        s.close()


def test_a_row_that_goes_again_is_counted_once(built_library):
    """HS_SAMPLE_APPEND_TOKEN and a row the bf16 kernel hands to the general one (more values outside
    its window than the side list holds): one token goes into the histogram, the one sampled."""
    from hydraserve_b200.engine import _device

    rows = 8
    logits = 5_000 + 64 * torch.randint(0, 4, (rows, VOCAB), generator=torch.Generator().manual_seed(2))
    logits = logits.cuda().bfloat16()
    s = _device.DeviceSampler("cuda:0", vocab_max=VOCAB, batch_max=rows, resident_slots=rows)
    try:
        params = [SamplingParams(temperature=2.0, seed=i, presence_penalty=0.5) for i in range(rows)]
        s.reset_slots(list(range(rows)))
        records, _ = s.run(logits, _device.pack_params(params, [0] * rows, list(range(rows))), append_token=True)
        assert not records["status"].any()
        assert [s.unique_count(i) for i in range(rows)] == [1] * rows
    finally:
        s.close()
