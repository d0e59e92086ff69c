"""Rows that start anywhere inside a 16-byte line: the same records as from an aligned copy (which
the parity tests hold against the checker), for every offset of the first token and for
vocabularies that leave zero to fourteen tokens outside the whole 16-byte chunks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from hydraserve_b200 import workloads  # noqa: E402

FIELDS = ("token", "status", "n_kept", "n_after_topk", "n_after_minp", "cut_bits", "n_cut_ties", "row_max", "log_z",
          "logprob", "n_top", "top_ids", "top_logprobs")


@pytest.mark.parametrize("vocab", [5, 4_099, 40_007, 70_000])
@pytest.mark.parametrize("offset", [0, 1, 2, 3, 4, 5, 6, 7])
def test_rows_at_every_offset_match_the_aligned_copy(built_library, vocab, offset):
    from hydraserve_b200.engine import _device

    w = workloads.config2(batch=8, vocab=vocab, seed=offset)
    w.logits[:4] = workloads.config3(batch=4, vocab=vocab, history_len=4, seed=offset).logits
    aligned = torch.from_numpy(w.logits.view(np.int16)).view(torch.bfloat16).cuda()
    stride = (vocab + 7 + 15) // 8 * 8
    room = torch.full((8, stride), 3.0e4, dtype=torch.bfloat16, device="cuda")  # (what lies outside a row must not count)
    room[:, offset:offset + vocab] = aligned
    s = _device.DeviceSampler("cuda:0", vocab_max=vocab, batch_max=8, resident_slots=8)
    try:
        want, _ = s.sample(aligned, w.histories, w.params, w.steps, None)
        got, _ = s.sample(room[:, offset:offset + vocab], w.histories, w.params, w.steps, None)
        for name in FIELDS:
            np.testing.assert_array_equal(got[name], want[name], err_msg=name)
        s.set_count_split(2)
        parts, _ = s.sample(room[:, offset:offset + vocab], w.histories, w.params, w.steps, None)
        np.testing.assert_array_equal(parts["token"], want["token"])
        np.testing.assert_array_equal(parts["n_kept"], want["n_kept"])
    finally:
        s.close()
