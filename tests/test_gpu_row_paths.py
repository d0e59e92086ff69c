"""The bf16 row kernel's rarer ways through a row against its usual ones: rows cut into parts, rows
of a batch of the stream and a little more or less, values spread over the whole range of a bf16,
masked rows; greedy rows at any address; and a step's records as the host puts them together."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from hydraserve_b200 import _lib  # noqa: E402
from hydraserve_b200.engine import SamplingParams, _device, sample_logits  # noqa: E402

COUNTS = ("status", "n_kept", "n_after_topk", "n_after_minp", "cut_bits", "n_cut_ties", "row_max")


@pytest.fixture(autouse=True)
def _lib_built(built_library):
    return built_library


def _sampler(vocab, batch):
    return _device.DeviceSampler("cuda:0", vocab_max=vocab, batch_max=batch, resident_slots=batch)


def _rows(kind, batch, vocab, seed=0):
    gen = torch.Generator().manual_seed(seed + vocab)
    x = torch.randn(batch, vocab, generator=gen) * 3
    if kind == "masked":           # all but a few hundred tokens are out
        x[:, torch.randperm(vocab, generator=gen)[: max(0, vocab - 300)]] = -float("inf")
    elif kind == "lowest":         # ... or at the type's lowest value
        x[:, torch.randperm(vocab, generator=gen)[: max(0, vocab - 300)]] = torch.finfo(torch.bfloat16).min
    elif kind == "wide":           # magnitudes from 1e-20 to 1e20
        x = torch.sign(x) * 10.0 ** (torch.rand(batch, vocab, generator=gen) * 40 - 20)
    elif kind == "few values":
        x = x.round()
    return x.to(torch.bfloat16).cuda()


# 16,384 tokens are the bound's sample and a batch of the stream, two of which are on their way at once
@pytest.mark.parametrize("vocab", [1, 7, 300, 4_096, 4_104, 16_384, 16_392, 32_768, 32_776, 36_864, 65_541, 151_936])
@pytest.mark.parametrize("kind", ["usual", "masked", "lowest", "wide", "few values"])
def test_small_top_k_rows_match_the_general_kernel(kind, vocab):
    """Both kernels finish such a row from its sorted candidates: the whole record is the same."""
    batch = 12
    logits = _rows(kind, batch, vocab)
    params = [SamplingParams(temperature=(0.7, 1.0, 1.3)[i % 3], top_k=min((1, 20, 50, 256)[i % 4], max(1, vocab - 1)), seed=i + 1, logprobs=5,
                             top_p=(1.0, 0.9)[i % 2], min_p=(0.0, 0.02)[i // 6],
                             **(dict(repetition_penalty=(1.2, 0.8)[i // 6], presence_penalty=0.5, frequency_penalty=0.3) if i % 5 else {}))
              for i in range(batch)]
    histories = [[(37 * j * j) % vocab for j in range(40 * i)] for i in range(batch)]
    s = _sampler(vocab, batch)
    try:
        with s.lock:
            slots = s.plan_slots(histories, params, vocab)
            rec = _device.pack_params(params, [2] * batch, slots)
            want, _ = s.run(logits, rec, general=True)
            for split in (0, 1, 2, 4):
                s.set_split(split)
                got, _ = s.run(logits, rec)
                for name in (*COUNTS, "token", "logprob", "n_top", "top_ids", "top_logprobs"):
                    np.testing.assert_array_equal(got[name], want[name], err_msg=f"{name}, {split} parts")
    finally:
        s.close()


# (47 tokens: parts without a chunk, and one of those has the loose tokens)
@pytest.mark.parametrize("vocab", [47, 8_192, 50_257, 65_543, 151_936])
@pytest.mark.parametrize("kind", ["usual", "few values", "masked"])
def test_a_counted_row_is_the_same_in_any_number_of_parts(kind, vocab):
    """The token too: it is the n-th member of a class whichever part holds it, and the same whether the
    class is looked up in the parts' lists or looked for in the whole row (rows off the 16-byte grid have
    members ahead of the first part)."""
    batch = 16
    room = torch.zeros((batch, vocab + 8 - vocab % 8), dtype=torch.bfloat16, device="cuda")
    logits = room[:, :vocab]  # (every row starts on a boundary; below, none does)
    logits.copy_(_rows(kind, batch, vocab))
    odd = torch.zeros((batch, room.shape[1] + 8), dtype=torch.bfloat16, device="cuda")[:, 3:3 + vocab]
    odd.copy_(logits)
    params = [SamplingParams(temperature=(0.4, 1.0, 1.4)[i % 3], top_p=(0.95, 0.7, 1.0)[i // 6], min_p=(0.0, 0.01)[i % 2], seed=11 * i + 1,
                             **(dict(repetition_penalty=1.1, frequency_penalty=0.2) if i % 4 else {})) for i in range(batch)]
    histories = [[(31 * j * j + i) % vocab for j in range(200 * i)] for i in range(batch)]
    s = _sampler(vocab, batch)
    try:
        with s.lock:
            slots = s.plan_slots(histories, params, vocab)
            for step in range(4):
                rec = _device.pack_params(params, [step] * batch, slots)
                s.set_count_split(1)
                want, _ = s.run(logits, rec)
                general, _ = s.run(logits, rec, general=True)
                for name in COUNTS:
                    np.testing.assert_array_equal(want[name], general[name], err_msg=f"{name}, against the general kernel")
                for split in (2, 3, 4, 5, 7, 8, 16, 0):
                    s.set_count_split(split)
                    for rows in (logits, odd):
                        got, _ = s.run(rows, rec)
                        for name in (*COUNTS, "token"):
                            np.testing.assert_array_equal(got[name], want[name], err_msg=f"{name}, {split} parts")
        # (a step knows which rows count, and cuts them as it sees fit)
        s.set_count_split(0)
        got = s.step(odd, histories, params, [3] * batch)
        assert [x.token_id for x in got] == want["token"].tolist()
    finally:
        s.close()


@pytest.mark.parametrize("vocab, parts", [(300_000, 2), (600_000, 4)])
def test_a_value_of_more_tokens_than_an_entry_holds(vocab, parts):
    """One value fills most of the first part, more tokens than one entry of a hand-over counts (131,070), and
    the 31 values above it, its neighbours in the count table, are drawn from: their members are looked up
    in a list that holds several entries of the full class.  (With 991 values below them the list has 32 x 32
    entries, and the search's first look goes to its last one.)"""
    batch, full, each = 32, 140_000, 20
    logits = torch.empty(batch, vocab, dtype=torch.bfloat16, device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(parts)
    for i in range(batch):
        low = torch.arange(vocab, device="cuda") % (991, 1_023, 1_055, 970 + i)[i % 4]  # (values from -1 down)
        x = (-0x4080 + low).to(torch.int16).view(torch.bfloat16)
        first = torch.randperm(vocab // parts, generator=gen, device="cuda")
        rest = torch.randperm(vocab - vocab // parts, generator=gen, device="cuda") + vocab // parts
        x[first[:full]] = 32.0
        for k in range(1, 32):
            x[first[full + each * k:full + each * (k + 1)]] = 32.0 + 0.25 * k
            x[rest[4 * each * k:4 * each * (k + 1)]] = 32.0 + 0.25 * k
        logits[i] = x
    params = [SamplingParams(temperature=2.0, seed=3 * i + 1) for i in range(batch)]
    s = _sampler(vocab, batch)
    s.set_token_draw(False)
    neighbours = 0
    try:
        with s.lock:
            for step in range(8):
                rec = _device.pack_params(params, [step] * batch, [-1] * batch)
                s.set_count_split(1)
                want, _ = s.run(logits, rec)
                s.set_count_split(parts)
                got, _ = s.run(logits, rec)
                for name in (*COUNTS, "token"):
                    np.testing.assert_array_equal(got[name], want[name], err_msg=name)
                neighbours += int((logits.cpu()[range(batch), want["token"]] > 32).sum())
    finally:
        s.close()
    assert neighbours > batch


def test_a_part_with_every_class_and_a_full_one():
    """Every value of the count table under every history count, and one of them more often than an entry
    counts: the longest list a part can hand over."""
    vocab, parts, batch = 600_000, 4, 6
    lowest, highest = 113 << 7, (113 << 7) + 3_072  # (raw bits of 2^-14 and 2^10)
    values = torch.arange(lowest, highest, dtype=torch.int16)
    values = torch.cat([values, values | -0x8000]).repeat(3)  # not in the history; there once; there twice
    gen = torch.Generator().manual_seed(3)
    raw = torch.full((batch, vocab), 0x4000, dtype=torch.int16)
    histories, per = [], vocab // parts
    for i in range(batch):
        here = torch.randperm(per, generator=gen)[:len(values)] + (0, parts - 1)[i % 2] * per
        elsewhere = torch.ones(vocab, dtype=torch.bool)
        elsewhere[(0, parts - 1)[i % 2] * per:][:per] = False
        raw[i, elsewhere] = torch.randint(lowest, highest, (vocab - per,), generator=gen, dtype=torch.int16)
        raw[i, here] = values
        once, twice = here[len(values) // 3:2 * len(values) // 3], here[2 * len(values) // 3:]
        histories.append(torch.cat([once, twice, twice]).tolist())
    logits = raw.view(torch.bfloat16).cuda()
    params = [SamplingParams(temperature=(1.0, 2.0)[i % 2], top_k=(3_000, 150_000, 400_000)[i // 2], seed=i + 1, frequency_penalty=0.01)
              for i in range(batch)]
    s = _sampler(vocab, batch)
    try:
        with s.lock:
            slots = s.plan_slots(histories, params, vocab)
            rec = _device.pack_params(params, [1] * batch, slots)
            s.set_count_split(1)
            want, _ = s.run(logits, rec)
            s.set_count_split(parts)
            for _ in range(3):
                got, _ = s.run(logits, rec)
                for name in (*COUNTS, "token"):
                    np.testing.assert_array_equal(got[name], want[name], err_msg=name)
    finally:
        s.close()


@pytest.mark.parametrize("penalised", [False, True])
@pytest.mark.parametrize("min_p", [1e-45, 1e-41, 3e-39, 1e-38, 5e-34, 2e-33, 1e-30, 0.05, 1.0])
def test_min_p_down_to_the_smallest_number(min_p, penalised):
    """Tens of thousands of tokens next to the maximum and as many far below it, every 0.002 of a score: where
    the threshold is a subnormal number or 0, tokens far below the line pass."""
    vocab, batch = 60_010, 6
    gen = torch.Generator().manual_seed(5)
    x = torch.randn(batch, vocab, generator=gen) * 0.01
    x[:3, -30_000:] = -torch.linspace(60, 125, 30_000)
    x[3:, -30_000:] = torch.tensor([-200.0, -99.0]).repeat(15_000)
    logits = x[:, torch.randperm(vocab, generator=gen)].to(torch.bfloat16).cuda()
    penalties = dict(repetition_penalty=1.2, frequency_penalty=0.3) if penalised else {}
    params = [SamplingParams(temperature=(1.0, 0.9)[i % 2], top_k=(0, 50_000, 0)[i % 3], min_p=min_p, seed=i, **penalties)
              for i in range(batch)]
    histories = [[(31 * j * j + i) % vocab for j in range(500)] for i in range(batch)]
    s = _sampler(vocab, batch)
    try:
        with s.lock:
            rec = _device.pack_params(params, [1] * batch, s.plan_slots(histories, params, vocab))
            want, _ = s.run(logits, rec, general=True)
            for split in (1, 3):
                s.set_count_split(split)
                got, _ = s.run(logits, rec)
                for name in COUNTS:
                    np.testing.assert_array_equal(got[name], want[name], err_msg=name)
    finally:
        s.close()


@pytest.mark.parametrize("counting, batch, vocab", [(1, 1, 131_072), (1, 1, 248_320), (1, 1, 262_144), (37, 37, 131_072),  # four to eight parts
                                                    (40, 120, 131_072), (20, 150, 151_936), (40, 160, 131_071),  # three; none
                                                    (64, 128, 131_072), (60, 75, 131_072), (4, 300, 131_072)])  # two; none
def test_the_parts_a_step_chooses(counting, batch, vocab):
    """A step knows which of its rows count and cuts them as it sees fit: the same rows whole."""
    logits = (torch.randn(batch, vocab, generator=torch.Generator(device="cuda").manual_seed(vocab), device="cuda") * 3).to(torch.bfloat16)
    params = [SamplingParams(temperature=1.0, top_p=0.95, seed=i, logprobs=3) if i % (batch // counting) == 0 and i < counting * (batch // counting)
              else SamplingParams(temperature=0.7, top_k=50, top_p=0.9, seed=i) for i in range(batch)]
    assert sum(p.top_k == 0 for p in params) == counting
    s = _sampler(vocab, batch)
    try:
        for step in range(3):
            s.set_count_split(1)
            want = s.step(logits, [[]] * batch, params, [step] * batch)
            s.set_count_split(0)
            assert s.step(logits, [[]] * batch, params, [step] * batch) == want
    finally:
        s.close()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("vocab", [1, 9, 31, 5_003, 50_257])
def test_greedy_rows_off_the_16_byte_grid(dtype, vocab):
    for offset in range(8):
        room = torch.full((5, vocab + 16), 3.0e4, dtype=dtype, device="cuda")  # (what lies outside a row must not count)
        rows = room[:, offset:offset + vocab]
        rows.copy_(torch.randn(5, vocab, generator=torch.Generator().manual_seed(offset)).to(dtype))
        rows[1] = 0.5                 # (the lowest id of a tie)
        rows[2, vocab - 1] = 9.0      # (the last token; the first)
        rows[3, 0] = 9.0
        got = sample_logits(rows, [[]] * 5, [SamplingParams()] * 5, steps=[0] * 5)
        want = [int((r == r.max()).nonzero()[0]) for r in rows.float().cpu()]
        assert [x.token_id for x in got] == want, offset


def test_mail_of_another_step_is_not_taken_for_this_one():
    """Rows with and without log-probabilities in turn, so that words of older steps stand in the mail;
    and the tags' way around: the step behind the last tag starts over with clean mail."""
    vocab, batch = 4_096, 6
    logits = _rows("usual", batch, vocab)
    s = _sampler(vocab, batch)
    try:
        for step, first in enumerate((None, 0xfffffffd, None, None, None, None)):
            if first is not None:
                _lib.check(s.lib, s.handle, s.lib.hs_debug_set(s.handle, 4, C.c_int(first - 2**32)), "hs_debug_set")
            params = [SamplingParams(temperature=1.0, top_k=(0, 40)[i % 2], seed=step * 10 + i, logprobs=3 if (i + step) % 2 else None)
                      for i in range(batch)]
            got = s.step(logits, [[]] * batch, params, [step] * batch)
            want, _ = s.sample(logits, [[]] * batch, params, [step] * batch)
            assert got == _device.records_to_samples(want, params, vocab)
    finally:
        s.close()
