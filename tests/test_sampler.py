"""The sampler's host side: the numbers of a request's stream, and which rows go to which kernel."""
import numpy as np
import pytest
import torch

from lightllm_b200 import SamplingParams
from lightllm_b200.sampling import sampler as S


@pytest.mark.parametrize("seed,request_id", [(42, 0), (0, 2 ** 63), (-1, 7)])
def test_numbers_drawn_ahead_are_those_drawn_one_by_one(seed, request_id):
    mask = 0xFFFF_FFFF_FFFF_FFFF
    one = np.random.Generator(np.random.Philox(key=np.array([seed & mask, request_id & mask], dtype=np.uint64)))
    stream = S.RequestStream(seed, request_id)
    assert [stream.uniform() for _ in range(3 * S.RequestStream.AHEAD + 5)] == \
        [float(one.random(dtype=np.float32)) for _ in range(3 * S.RequestStream.AHEAD + 5)]


@pytest.mark.parametrize("temperatures,kernel", [([0.0, 9e-6], "argmax"), ([0.0, 1e-5], "sample"), ([0.0, float("nan")], "sample"),
                                                 ([float("nan"), 0.0], "sample"), ([], "argmax")])
def test_only_rows_that_are_all_greedy_go_to_the_argmax(monkeypatch, temperatures, kernel):
    calls = []
    monkeypatch.setattr(S.ops, "argmax", lambda logits, out: calls.append("argmax"))
    monkeypatch.setattr(S.ops, "sample", lambda *args: calls.append("sample"))
    params = [SamplingParams(temperature=t) for t in temperatures]
    assert all(p.greedy for p in params) == (kernel == "argmax")
    S.Sampler(torch.device("cpu")).sample_device(torch.zeros(len(params), 8), list(range(len(params))), params)
    assert calls == [kernel]
