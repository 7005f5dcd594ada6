"""The sampling kernel's thresholds over long rows where its bins are of no use or at their edges: ties, masked values, values that are
not numbers, the smallest and largest k and p."""
import numpy as np
import pytest
import torch

from tests.plain.qwen2_plain import plain_draw, plain_sampling_probs
from tests.test_kernels_gpu import dev, ops  # noqa: F401

pytestmark = pytest.mark.gpu


def rows(kind, V, g):
    x = torch.randn(V, generator=g) * 3.0
    if kind == "equal":
        x = torch.full((V,), 1.25)
    elif kind == "two":                  # a few high values, thousands of equal low ones: the threshold lies among the ties
        x = torch.where(torch.arange(V) % 1000 == 7, 4.0, -1.0)
    elif kind == "masked":
        x[torch.rand(V, generator=g) < 0.999] = -float("inf")
    elif kind == "wide":                 # most values below the last bin
        x = x * 40.0
    elif kind == "narrow":               # all values in one bin
        x = x * 1e-4
    return x


@pytest.mark.parametrize("V", [8192, 30011, 151936])
@pytest.mark.parametrize("kind", ["normal", "equal", "two", "masked", "wide", "narrow"])
def test_thresholds(ops, kind, V):  # noqa: F811
    g = torch.Generator().manual_seed(V)
    x = rows(kind, V, g)
    filters = [(1, 1.0), (5, 1.0), (40, 0.9), (V - 1, 1.0), (0, 0.5), (0, 0.999), (0, 1e-6), (300, 0.3)]
    us = [0.02, 0.37, 0.71, 0.98]
    many = [(k, p, u) for k, p in filters for u in us]
    f = lambda v, dt=torch.float32: torch.tensor(v, dtype=dt, device=dev())  # noqa: E731
    out = torch.empty(len(many), dtype=torch.int32, device=dev())
    ops.sample(x[None].repeat(len(many), 1).contiguous().to(dev()), f([0.8] * len(many)), f([m[0] for m in many], torch.int32),
               f([m[1] for m in many]), f([0.0] * len(many)), f([m[2] for m in many]), out)
    for (k, p, u), got in zip(many, out.tolist()):
        probs = plain_sampling_probs(x.numpy(), 0.8, k, p, 0.0)
        if p < 1.0 and kind in ("equal", "two", "narrow"):
            # the kernel keeps all of a tie (or, where rounding decides, of what is within it of one); the plain filter a part
            probs = plain_sampling_probs(x.numpy(), 0.8, k, 1.0, 0.0)
            assert probs[got] > 0.0
            continue
        assert probs[got] > 0.0, (k, p, u)
        want = plain_draw(probs, u)
        if got != want:          # float sums of V terms against float64: the draw lies that close to a boundary
            cdf = np.cumsum(probs)
            assert min(abs(cdf[min(got, want)] - u), abs(cdf[max(got, want) - 1] - u)) < 1e-4, (k, p, u)


def test_rows_that_are_not_numbers(ops):  # noqa: F811
    V = 20000
    x = torch.randn(3, V, generator=torch.Generator().manual_seed(3))
    x[0, 11] = float("nan")
    x[1, 17] = float("inf")
    x[2] = float("nan")
    out = torch.empty(3, dtype=torch.int32, device=dev())
    f = lambda v, dt=torch.float32: torch.full((3,), v, dtype=dt, device=dev())  # noqa: E731
    ops.sample(x.to(dev()), f(1.0), f(50, torch.int32), f(0.9), f(0.0), f(0.4), out)
    assert all(0 <= t < V for t in out.tolist())


@pytest.mark.parametrize("V", [2000, 8192, 151936])          # one block a row; a cluster of blocks
def test_zeros_of_both_signs(ops, V):  # noqa: F811
    """+0 lies above -0 in the order that top-k goes by: a k-th place among zeros keeps the same tokens at every launch."""
    x = torch.full((V,), -30.0)
    plus, minus = [200, 901, 1500], [17, 300, 1999]
    x[100], x[plus], x[minus] = 1.0, 0.0, -0.0
    us = [(i + 0.5) / 40 for i in range(40)]
    many = [(k, u) for k in (2, 3, 4, 5, 6, 7) for u in us]
    f = lambda v, dt=torch.float32: torch.tensor(v, dtype=dt, device=dev())  # noqa: E731
    rows_ = x[None].repeat(len(many), 1).contiguous().to(dev())
    out = torch.empty(len(many), dtype=torch.int32, device=dev())
    args = f([1.0] * len(many)), f([m[0] for m in many], torch.int32), f([1.0] * len(many)), f([0.0] * len(many)), f([m[1] for m in many])
    for _ in range(20):
        ops.sample(rows_, *args, out)
        got = out.tolist()
        for k in (2, 3, 4, 5, 6, 7):
            kept = sorted([100] + plus + (minus if k > 1 + len(plus) else []))
            mass = np.cumsum([np.e if i == 100 else 1.0 for i in kept])
            want = [kept[int(np.searchsorted(mass, u * mass[-1]))] for u in us]
            assert got[: len(us)] == want, k
            got = got[len(us):]
