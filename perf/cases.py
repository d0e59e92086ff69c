"""The sampler's work as its users have it done: one case per way the per-step sampler is called
in a serving process, over the sizes and options those calls come in.

    listed()               the named cases
    draw(rng)              one more case of the same ranges
    prepare(case, seed)    what the caller has in hand before the call
    run(state)             one call through the public entry points, and its outputs
    work(case)             bytes and operations the call cannot do without
    tolerance(case)        how far another correct implementation's outputs may be off

A case is a dict of plain values:

    call      "serve"    sample_logits with request ids: the decode step of a serving loop whose token
                         histograms stay on the device; the history of every request has grown by one
                         token since its last step
              "packed"   the same step with the result as one record array (a worker's reply)
              "drop_in"  sample_logits as the reference's callers write it, full histories every step
              "chained"  DeviceSampler.launch: parameters, records and sampled ids stay on the device
              "sharded"  sample_logits_sharded on one rank's slice of the vocabulary
    batch, vocab, dtype  shape and type of the logits
    mix       the requests' parameters and the shape of their logits, see _requests
    penalties whether the requests use repetition / presence / frequency penalties
    history   longest history, in tokens (prompt and generated)
    logprobs  log-probabilities asked for per row, -1 for none

Integer results (token ids, candidate counts) do not depend on the order of any sum in this
sampler and are compared exactly; log-probabilities are 32-bit floats.
"""
import itertools
import math

import numpy as np
import torch

from hydraserve_b200 import _lib
from hydraserve_b200.engine import SamplingParams, sample_logits, sample_logits_packed
from hydraserve_b200.engine import _device
from hydraserve_b200.engine.sharded import sample_logits_sharded

MOST_TOKENS = 1024 * 151_936   # logits of the largest listed call
MOST_HISTORY = 256 * 32_768    # history tokens of the largest listed call
CHAIN = 16                     # parameter sets a chained loop has on the device


def _case(call, batch, vocab, dtype="bf16", mix="chat", penalties=True, history=0, logprobs=-1):
    return {"call": call, "batch": batch, "vocab": vocab, "dtype": dtype, "mix": mix,
            "penalties": penalties, "history": history, "logprobs": logprobs}


def listed():
    cases = [
        # the default request (temperature 0) with one stream running: the smallest call there is
        ("greedy_1", _case("serve", 1, 151_936, mix="greedy", penalties=False)),
        # a full default batch of the same
        ("greedy_64", _case("serve", 64, 248_320, mix="greedy", penalties=False)),
        # one interactive user with the usual settings: per-token latency
        ("chat_1", _case("serve", 1, 151_936, mix="chat", history=512)),
        # first token after a prefill: batch 1, the prompt as the history, nothing resident
        ("first_token", _case("drop_in", 1, 248_320, mix="nucleus", history=8_192)),
        # the reference's CPU-runnable check: fp32 logits, one greedy row, three chat rows
        ("fp32_check_4", _case("drop_in", 4, 151_936, dtype="f32", mix="check", history=256)),
        # the fp32-logits serving mode with requests that set top_p alone
        ("fp32_nucleus_32", _case("serve", 32, 151_936, dtype="f32", mix="nucleus", history=2_048)),
        # a decode step of mixed requests with 20 log-probabilities each, replied as one array
        ("decode_packed_64", _case("packed", 64, 151_936, mix="decode", history=4_096, logprobs=20)),
        # the same requests from a caller that knows no request ids, at an odd vocabulary and batch
        ("drop_in_odd_33", _case("drop_in", 33, 50_257, mix="decode", history=4_096, logprobs=5)),
        # large-vocabulary stress: near-flat and peaked rows, all penalties, long histories
        ("stress_256", _case("serve", 256, 248_320, mix="stress", history=32_768)),
        # the largest step: a thousand requests with parameters of every kind
        ("random_1024", _case("serve", 1_024, 151_936, mix="random", history=8_192)),
        # a decode loop that never leaves the device
        ("chained_256", _case("chained", 256, 248_320, mix="stress", penalties=False)),
        # one rank's share of a vocabulary split over eight
        ("sharded_128", _case("sharded", 128, 31_040, mix="shard", penalties=False, logprobs=20)),
    ]
    return [dict(case, name=name) for name, case in cases]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """A call of a kind listed above at sizes from all over the range: batches of 1 to 1,024,
    vocabularies of 16,000 to 262,144 (odd ones too), histories of 16 to 32,768 tokens."""
    call = rng.choice(["serve", "serve", "serve", "packed", "drop_in", "drop_in", "chained", "sharded"])
    if call == "sharded":
        vocab = _log_uniform(rng, 8_000, 131_072) & ~7
        batch = _log_uniform(rng, 1, 512)
        return _case(call, batch, vocab, mix="shard", penalties=False, logprobs=rng.choice([-1, 5, 20]))
    vocab = _log_uniform(rng, 16_000, 262_144)
    if rng.random() < 0.75:
        vocab &= ~63  # most heads are padded; the rest stay as odd as they came
    dtype = "f32" if rng.random() < 0.25 else "bf16"
    mix = rng.choice(["greedy", "chat", "check", "nucleus", "decode", "stress", "random"])
    most = 64 if dtype == "f32" else 1_024
    batch = _log_uniform(rng, 1, min(most, MOST_TOKENS // vocab))
    penalties = mix != "greedy" and call != "chained" and rng.random() < 0.75
    history = 0
    if penalties:
        history = _log_uniform(rng, 16, min(32_768, MOST_HISTORY // batch))
        if call == "drop_in":
            history = max(16, min(history, 300_000 // batch))
    logprobs = -1
    if mix != "greedy" and rng.random() < 0.4:
        logprobs = rng.choice([0, 1, 5, 20])
    return _case(call, batch, vocab, dtype, mix, penalties, history, logprobs)


def _requests(case, rng):
    """Per row the request's parameters and the spread of its logits."""
    params, spread = [], []
    for i in range(case["batch"]):
        p = {"seed": 1 + int(rng.integers(2**40))}
        if case["logprobs"] >= 0:
            p["logprobs"] = case["logprobs"]
        sigma, mix = 3.0, case["mix"]
        if mix == "decode":    # greedy, top_p, top_k + min_p, top_k + top_p in turn
            mix = ("greedy", "nucleus", "top_k_min_p", "top_k_top_p")[i % 4]
            if case["penalties"]:
                p.update(presence_penalty=0.5, frequency_penalty=0.3)
        elif mix == "check":   # one greedy row, the others like a chat request
            mix, sigma = ("chat" if i else "greedy"), 2.5
            if case["penalties"] and i:
                p.update(repetition_penalty=1.1)
        elif mix == "stress":  # half near-flat rows of which top_p keeps tens of thousands, half peaked
            mix, sigma = ("flat", 0.1) if i < case["batch"] // 2 else ("peaked", 4.0)
            if case["penalties"]:
                p.update(repetition_penalty=1.05, presence_penalty=0.4, frequency_penalty=0.2)
        elif mix == "random":
            if case["penalties"]:
                p.update(repetition_penalty=1.0 + rng.uniform(0, 0.6), presence_penalty=rng.uniform(0, 0.6),
                         frequency_penalty=rng.uniform(0, 0.6))
        elif mix == "nucleus":
            if case["penalties"]:
                p.update(presence_penalty=0.5, frequency_penalty=0.3)
        elif mix == "chat":
            if case["penalties"]:
                p.update(repetition_penalty=1.1)
        if mix == "chat":
            p.update(temperature=0.7, top_k=50, top_p=0.9)
        elif mix == "nucleus":
            p.update(temperature=1.0, top_p=0.95)
        elif mix == "top_k_min_p":
            p.update(temperature=1.0, top_k=20, min_p=0.05)
        elif mix == "top_k_top_p":
            p.update(temperature=1.2, top_k=40, top_p=0.8)
        elif mix == "flat":
            p.update(temperature=1.0, top_p=0.99)
        elif mix == "peaked":
            p.update(temperature=1.0, top_k=50, top_p=0.9, min_p=0.02)
        elif mix == "random":
            p.update(temperature=rng.uniform(0.3, 1.5), top_k=int(rng.choice([0, 20, 50, 200])),
                     top_p=rng.uniform(0.7, 1.0), min_p=float(rng.choice([0.0, 0.05])))
        elif mix == "shard":
            p.update(temperature=0.8, top_k=50, top_p=0.9)
        params.append(SamplingParams(**p))
        spread.append(sigma)
    return params, spread


def _lengths(case, rng):
    """Tokens in each request's history: the longest for the shapes whose requests are alike,
    else anything up to it."""
    longest = case["history"]
    if longest == 0 or case["mix"] in ("stress", "check", "chat") or case["batch"] == 1:
        return [longest] * case["batch"]
    low = longest // 16 if case["mix"] == "random" else 1
    return [int(n) for n in rng.integers(max(1, low), longest + 1, case["batch"])]


def _histories(case, lengths, seed, device):
    """Token ids, uniform over the vocabulary, or bounded power-law (a few ids very often) for
    the mixed decode requests; Python lists of ints, as a serving loop keeps them."""
    gen = torch.Generator(device=device).manual_seed(seed)
    total, vocab = sum(lengths), case["vocab"]
    u = torch.rand(max(total, 1), generator=gen, device=device, dtype=torch.float64)
    if case["mix"] == "decode":
        ids = (1.0 - u * (1.0 - float(vocab + 1) ** -0.1)) ** -10.0 - 1.0
    else:
        ids = u * vocab
    ids = ids.long().clamp_(0, vocab - 1).cpu().tolist()
    out, at = [], 0
    for n in lengths:
        out.append(ids[at:at + n])
        at += n
    return out


_serial = itertools.count()


class State:
    pass


def prepare(case, seed):
    device = torch.device("cuda", torch.cuda.current_device())
    rng = np.random.default_rng(seed)
    batch, vocab = case["batch"], case["vocab"]
    s = State()
    s.case = case
    s.params, spread = _requests(case, rng)
    gen = torch.Generator(device=device).manual_seed(seed)
    dtype = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
    s.logits = torch.empty((batch, vocab), dtype=dtype, device=device)
    for i in range(0, batch, 64):  # (in pieces: the fp32 values of a large batch need not exist at once)
        part = torch.randn((min(64, batch - i), vocab), generator=gen, device=device)
        s.logits[i:i + 64] = part * torch.tensor(spread[i:i + 64], device=device)[:, None]
    s.histories = _histories(case, _lengths(case, rng), seed + 1, device)
    s.steps = [int(n) for n in rng.integers(0, 2_048, batch)]
    s.ids = None
    if case["call"] == "chained":
        # the loop's own sampler and buffers, and the parameters of its next steps
        s.sampler = _device.DeviceSampler(device, vocab_max=vocab, batch_max=batch, resident_slots=batch, hist_cap=4_096)
        s.d_params = []
        for t in range(CHAIN):
            rec = _device.pack_params(s.params, [n + t for n in s.steps], [-1] * batch)
            s.d_params.append(torch.from_numpy(rec.view(np.uint8).reshape(batch, -1).copy()).to(device))
        s.d_out = torch.zeros((batch, _lib.ROW_OUT.itemsize), dtype=torch.uint8, device=device)
        s.tokens = torch.zeros(batch, dtype=torch.int32, device=device)
        s.at = 0
    else:
        # the process's sampler, sized for more live requests than one step decodes
        _device.sampler_for(device, vocab, 4 * batch, max(case["history"], 1))
    if case["call"] in ("serve", "packed"):
        # requests in flight: the token each one gains per step, and a first step behind them
        s.ids = [("request", next(_serial)) for _ in range(batch)]
        s.token_at = rng.integers(0, vocab, batch)
        s.token_by = rng.integers(1, vocab, batch)
        if case["penalties"]:
            sample_logits_packed(s.logits, s.histories, s.params, steps=s.steps, request_ids=s.ids)
    return s


def _grow(s):
    """Every request has generated one more token since its last step."""
    s.steps = [n + 1 for n in s.steps]
    if s.case["penalties"]:
        s.token_at = (s.token_at + s.token_by) % s.case["vocab"]
        for history, token in zip(s.histories, s.token_at.tolist()):
            history.append(token)


def _of_tuple(s, samples):
    out = {"token": np.array([x.token_id for x in samples])}
    if s.case["logprobs"] >= 0:
        out["logprob"] = np.array([x.logprob for x in samples], dtype=np.float32)
        top = [x.top_logprobs for x in samples]
        out["top_id"] = np.array([[t[0] for t in row] for row in top], dtype=np.int64)
        out["top_logprob"] = np.array([[t[1] for t in row] for row in top], dtype=np.float32)
    return out


def _of_records(s, packed):
    records = packed.records
    out = {"token": packed.token_ids}
    if s.case["mix"] != "greedy":
        for name in ("n_kept", "n_after_topk", "n_after_minp", "cut_bits", "status", "row_max"):
            out[name] = records[name]
    if s.case["logprobs"] >= 0:
        there = np.arange(_lib.HS_MAX_LOGPROBS) < records["n_top"][:, None]
        out["logprob"], out["n_top"] = records["logprob"], records["n_top"]
        out["top_id"] = np.where(there, records["top_ids"], -1)
        out["top_logprob"] = np.where(there, records["top_logprobs"], np.float32(0))
    return out


def run(s):
    call = s.case["call"]
    if call == "chained":
        s.at = (s.at + 1) % CHAIN
        s.sampler.launch(s.logits, s.d_params[s.at], s.d_out, tokens_out=s.tokens)
        words = s.d_out.view(torch.int32)
        return {"token": s.tokens, "counts": words[:, 3:10], "row_max": s.d_out.view(torch.float32)[:, 10]}
    if call == "sharded":
        return _of_tuple(s, sample_logits_sharded(s.logits, s.histories, s.params, steps=s.steps, vocab_offset=0,
                                                  vocab_total=s.case["vocab"]))
    if call == "drop_in":
        return _of_tuple(s, sample_logits(s.logits, s.histories, s.params, steps=s.steps))
    _grow(s)
    if call == "packed":
        return _of_records(s, sample_logits_packed(s.logits, s.histories, s.params, steps=s.steps, request_ids=s.ids))
    return _of_tuple(s, sample_logits(s.logits, s.histories, s.params, steps=s.steps, request_ids=s.ids))


def work(case):
    """The logits once; of the history the ids (drop-in calls) or the resident (id, count) pairs, at
    most one per vocabulary entry; parameters and records.  One operation per logit."""
    tokens = case["batch"] * case["vocab"]
    average = case["history"] if case["mix"] in ("stress", "check", "chat") else case["history"] / 2
    seen = case["batch"] * (4 * average if case["call"] == "drop_in" else 8 * min(average, case["vocab"]))
    rows = case["batch"] * (_lib.ROW_PARAMS.itemsize + _lib.ROW_OUT.itemsize)
    return {"bytes": tokens * (2 if case["dtype"] == "bf16" else 4) + seen + rows, "flops": tokens}


def tolerance(case):
    # sums of 2**-40 units behind a 32-bit logarithm; token ids and counts have no room to differ
    return {"rel": 1e-5, "max": 1e-4, "differ": 0.0}
