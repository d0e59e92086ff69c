"""The native host side of a step against a stand-in for the CUDA library that notes what each step
asks of it; no GPU needed."""
import ctypes as C
import importlib.util
import subprocess
import sysconfig
import threading
from types import SimpleNamespace

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from hydraserve_b200 import _lib, build  # noqa: E402
from hydraserve_b200.engine import SamplingParams, TokenSample, _device  # noqa: E402

VOCAB = 1_000


class _Desc(C.Structure):
    _fields_ = [(n, C.c_size_t) for n in ("bytes", "resets_at", "slots_at", "offsets_at", "tokens_at")] + \
               [(n, C.c_int32) for n in ("n_resets", "n_appends", "max_tokens", "repeats")]


class Library:
    """What the stepper calls, by address.  `steps` has (resets, {slot: tokens}) per step;
    `status` is what the next hs_step answers."""

    def __init__(self):
        self.steps, self.status, self.calls = [], 0, 0
        self.block, self.text = C.create_string_buffer(1 << 16), C.create_string_buffer(b"as asked for")
        self.records = np.zeros(64, dtype=_lib.ROW_OUT)
        self.ids = np.zeros(64, dtype=np.int32)
        p, pp, i = C.c_void_p, C.POINTER(C.c_void_p), C.c_int
        self.entries = [C.CFUNCTYPE(i, p, C.c_size_t, pp)(self._block),
                        C.CFUNCTYPE(i, p, p, i, C.c_int64, i, i, C.POINTER(_Desc), pp, p)(self._step),
                        C.CFUNCTYPE(i, p, p, i, C.c_int64, i, i, pp, p)(self._greedy),
                        C.CFUNCTYPE(i, p, p)(self._wait),
                        C.CFUNCTYPE(p, p)(lambda h: C.addressof(self.text))]

    def stepper(self, host, book, base=100):
        return host.Stepper(1, book, base, _lib.SamplerError, *(C.cast(f, C.c_void_p).value for f in self.entries))

    def _block(self, h, n, out):
        self.calls += 1
        out[0] = C.addressof(self.block)
        return 0

    def _step(self, h, logits, dtype, stride, batch, vocab, desc, out, stream):
        self.calls += 1
        d = desc[0]
        ints = lambda at, n: np.frombuffer(self.block, np.int32, n, at).tolist()  # noqa: E731
        offsets = ints(d.offsets_at, d.n_appends + 1) if d.n_appends else [0]
        tokens = ints(d.tokens_at, offsets[-1])
        slots = ints(d.slots_at, d.n_appends)
        self.steps.append((ints(d.resets_at, d.n_resets),
                           {s: tokens[a:b] for s, a, b in zip(slots, offsets, offsets[1:])}))
        out[0] = self.records.ctypes.data
        return self.status

    def _greedy(self, h, logits, dtype, stride, batch, vocab, out, stream):
        self.calls += 1
        out[0] = self.ids.ctypes.data
        return 0

    def _wait(self, h, stream):
        return 0


class Sampler:
    def __init__(self, n_slots=4, host=_device._host):
        self.library = Library()
        self.book = host.SlotBook(n_slots)
        self.host = self.library.stepper(host, self.book)
        self.params = SamplingParams(temperature=1.0, seed=1, presence_penalty=0.5)

    def step(self, requests, steps=None):
        """One step of {request: history}; (resets, appends) as the library got them."""
        n = len(requests)
        self.host.step(0, 1, VOCAB, VOCAB, list(requests.values()), [self.params] * n, steps or [0] * n, list(requests), 0, False)
        return self.library.steps[-1]

    def slot(self, request):
        return self.book.entries[request][0]


def _bad_token(s, requests):
    with pytest.raises((TypeError, ValueError)):
        s.step({**requests, "bad": [1, "no token"]})


def _bad_step(s, requests):
    with pytest.raises((TypeError, ValueError)):
        s.step(requests, [0] * (len(requests) - 1) + [None])


def _bad_library(s, requests):
    s.library.status = -3
    with pytest.raises(_lib.SamplerError, match="as asked for"):
        s.step(requests)
    s.library.status = 0


@pytest.mark.parametrize("fail", [_bad_token, _bad_step, _bad_library])
@pytest.mark.parametrize("history", [[], [5]])
def test_a_request_of_a_failed_step_starts_over(fail, history):
    """A failed step may not have emptied the histograms it was to empty: the next step must ask for it
    again, for a new request in another's place and for one whose history shrank, with and
    without tokens of their own."""
    s = Sampler(n_slots=3)
    assert s.step({"a": [1, 2, 3]}) == ([0], {0: [1, 2, 3]})
    s.book.release("a")
    fail(s, {"b": history})  # (takes the slot that holds a's tokens)
    resets, appends = s.step({"b": [*history, 7]})
    assert resets == [s.slot("b")] and appends == {s.slot("b"): [*history, 7]}
    fail(s, {"b": history[:-1]})
    resets, appends = s.step({"b": [8, 9]})
    assert resets == [s.slot("b")] and appends == {s.slot("b"): [8, 9]}


@pytest.mark.parametrize("tokens", [[1, "no token"], [1, 2]])
def test_a_plan_that_does_not_reach_the_device_is_forgotten(tokens):
    """The same where plan and device calls are apart (DeviceSampler.plan_slots)."""
    book, calls = _device.SlotBook(4), []

    def append(slots, arrays, vocab):
        if tokens == [1, 2]:
            raise _lib.SamplerError("as asked for")
        [np.asarray(a, dtype=np.int64) for a in arrays]
        calls.append((slots, [list(a) for a in arrays]))

    fake = SimpleNamespace(book=book, scratch_base=100, reset_slots=lambda slots: calls.append(list(slots)), append_tokens=append)
    params = [SamplingParams(temperature=1.0, seed=1, presence_penalty=0.5)] * 2
    with pytest.raises((TypeError, ValueError, _lib.SamplerError)):
        _device.DeviceSampler.plan_slots(fake, [[], tokens], params, VOCAB, ["a", "b"])
    assert not dict(book.entries)
    calls.clear()
    fake.append_tokens = lambda slots, arrays, vocab: calls.append((slots, [list(a) for a in arrays]))
    slots = _device.DeviceSampler.plan_slots(fake, [[4], [5]], params, VOCAB, ["a", "b"])
    assert calls == [slots, (slots, [[4], [5]])]


def test_a_step_on_a_closed_sampler_fails_without_a_call():
    s = Sampler()
    s.step({"a": [1]})
    destroyed = []
    sampler = object.__new__(_device.DeviceSampler)
    sampler.handle, sampler.host, sampler.lock = C.c_void_p(1), s.host, threading.RLock()
    sampler.lib = SimpleNamespace(hs_destroy=destroyed.append)
    sampler.close()
    sampler.close()
    assert len(destroyed) == 1
    calls = s.library.calls
    with pytest.raises(_lib.SamplerError):
        s.step({"a": [1, 2]})
    with pytest.raises(_lib.SamplerError):
        s.host.greedy(0, 1, VOCAB, 2, VOCAB, 0, False)
    assert s.library.calls == calls


@pytest.mark.parametrize("named", ["cuda", "cuda:0", 0, torch.device("cuda"), torch.device("cuda:0")])
def test_a_gpu_has_one_sampler_however_it_is_named(monkeypatch, named):
    made, released = [], []

    class Fake:
        hist_cap, users, retired = VOCAB, 0, False

        def __init__(self, device, vocab_max, batch_max, **_):
            self.device, self.vocab_max, self.batch_max = device, vocab_max, batch_max
            self.release_request = released.append
            made.append(device)

    monkeypatch.setattr(_device, "DeviceSampler", Fake)
    monkeypatch.setattr(_device, "_samplers", {})
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    first = _device.sampler_for(named, VOCAB, 4)
    for other in ("cuda", "cuda:0", 0, torch.device("cuda"), torch.device("cuda:0")):
        assert _device.sampler_for(other, VOCAB, 4) is first
        _device.release_request("a", other)
    assert made == [torch.device("cuda:0")] and released == ["a"] * 5


@pytest.mark.parametrize("batched", ["1", "0"])
@pytest.mark.parametrize("params", [SamplingParams(), SamplingParams(temperature=1.0, seed=1)])
def test_a_step_that_is_no_number_is_refused_before_anything_else(monkeypatch, params, batched):
    """(the reference's int(step) for every row, plain greedy ones too)"""
    from hydraserve_b200.engine import sample_logits, sample_logits_packed

    monkeypatch.setenv("HYDRASERVE_BATCHED_GREEDY", batched)
    monkeypatch.setattr(_device, "_target_device", lambda logits: pytest.fail("the call went on"))
    for call in (sample_logits, sample_logits_packed):
        for step, error in ((None, TypeError), ("three", ValueError), ([1], TypeError)):
            with pytest.raises(error):
                call(torch.zeros(2, 5), [[], []], [params] * 2, steps=[0, step])
    assert _device.longest_history([[], []], [params] * 2, [2.5, True]) == (-1 if params == SamplingParams() else 0)


def test_the_extension_is_built_for_this_interpreter():
    assert _device._host.__file__ == str(build.HOST_OUTPUT)
    assert build.HOST_OUTPUT.name == "_host" + sysconfig.get_config_var("EXT_SUFFIX")


def test_histories_read_the_same_without_the_interpreters_compact_ints(tmp_path):
    """The form older interpreters get, built beside the other."""
    path = tmp_path / build.HOST_OUTPUT.name
    subprocess.run(["g++", *build.CXX_FLAGS, "-DHS_COMPACT_INTS=0", "-I", sysconfig.get_paths()["include"],
                    "-o", str(path), *map(str, build.HOST_SOURCES)], check=True)
    spec = importlib.util.spec_from_file_location("_host", path)
    other = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(other)
    other.bind(TokenSample, _device._as_int64, _device.draw_unseeded_keys)
    history = [0, 5, VOCAB - 1, VOCAB, -1, -2**31, 2**31, 2**40, 2**62, -2**63, 7]
    want = [0, 5, VOCAB - 1, -1, -1, -1, -1, -1, -1, -1, 7]
    for host in (_device._host, other):
        s = Sampler(host=host)
        assert s.step({"a": history, "b": tuple(history)})[1] == {s.slot("a"): want, s.slot("b"): want}
        with pytest.raises(OverflowError):
            s.step({"a": [*history, 2**63]})


@pytest.mark.parametrize("defines,word", [([], "ia32_pause"), (["-U__x86_64__", "-D__aarch64__"], "yield"), (["-U__x86_64__"], None)])
def test_the_wait_hint_is_the_hosts_own(defines, word):
    header = build.PKG / "csrc" / "hs_pause.h"
    text = subprocess.run(["g++", "-E", "-P", "-x", "c++", *defines, str(header)], check=True, capture_output=True, text=True).stdout
    assert [w for w in ("ia32_pause", "yield") if w in text] == ([word] if word else [])
