"""The sampling kernel's thresholds over long rows where its bins are of no use or at their edges: ties, masked values, values that are
not numbers, the smallest and largest k and p."""
import numpy as np
import pytest
import torch

from tests.plain.qwen2_plain import plain_sampling_probs
from tests.test_kernels_gpu import dev, ops  # noqa: F401

pytestmark = pytest.mark.gpu


def rows(kind, V, g):
    x = torch.randn(V, generator=g) * 3.0
    if kind == "equal":
        x = torch.full((V,), 1.25)
    elif kind == "two":                  # a few high values, thousands of equal low ones: the threshold lies among the ties
        x = torch.where(torch.arange(V) % 1000 == 7, 4.0, -1.0)
    elif kind == "halves":               # two values in no order
        x = torch.where(torch.rand(V, generator=g) < 0.5, 0.75, 0.25)
    elif kind == "grid":                 # values of 8 bits: hundreds of ties at every one
        x = x.bfloat16().float()
    elif kind == "masked":
        x[torch.rand(V, generator=g) < 0.999] = -float("inf")
    elif kind == "far":                  # a mask of large numbers: nearly all values share the last bin
        x[torch.rand(V, generator=g) < 0.999] = -1e9
    elif kind == "wide":                 # most values below the last bin
        x = x * 40.0
    elif kind == "flat":
        x = x * 0.01
    elif kind == "narrow":               # floats next to one another
        x = x * 1e-4
    return x


def kept(x, temperature, k, p):
    """Masses of the tokens that stay, all ties among them, in float64 from the scaled float32 logits, and which part of the mass
    the rounding of an exponential (a few ulps at the threshold) may add or leave out."""
    s = x.numpy() * (np.float32(1.0) / np.float32(temperature))
    e = np.exp((s - s.max()).astype(np.float64))
    if 0 < k < len(s):
        e[s < np.sort(s)[-k]] = 0.0
    if p >= 1.0:
        return e, 0.0
    f = e.astype(np.float32)
    order = np.argsort(-f, kind="stable")
    mass = np.cumsum(e[order])
    t = f[order[np.searchsorted(mass, p * mass[-1] * (1 - 1e-12))]]
    edge = (f != t) & (np.abs(f.astype(np.float64) / t - 1.0) < 4e-7)
    return np.where(f >= t, e, 0.0), float(e[edge].sum() / e[f >= t].sum())


# a cluster's rows from the shortest on; the longest that its shared memory holds, and the next, which one block takes
@pytest.mark.parametrize("kind,V", [(k, V) for V in (8192, 30011, 151936)
                                    for k in ("normal", "equal", "two", "halves", "grid", "masked", "far", "wide", "flat", "narrow")]
                         + [("normal", 430001), ("grid", 442368), ("normal", 442369)])
def test_thresholds(ops, kind, V):  # noqa: F811
    g = torch.Generator().manual_seed(V)
    x = rows(kind, V, g)
    filters = [(1, 1.0), (5, 1.0), (40, 0.9), (V - 1, 1.0), (0, 0.5), (0, 0.999), (0, 1e-6), (300, 0.3), (V // 2, 0.7)]
    us = [0.02, 0.37, 0.71, 0.98]
    many = [(k, p, u) for k, p in filters for u in us]
    f = lambda v, dt=torch.float32: torch.tensor(v, dtype=dt, device=dev())  # noqa: E731
    out = torch.empty(len(many), dtype=torch.int32, device=dev())
    ops.sample(x[None].repeat(len(many), 1).contiguous().to(dev()), f([0.8] * len(many)), f([m[0] for m in many], torch.int32),
               f([m[1] for m in many]), f([0.0] * len(many)), f([m[2] for m in many]), out)
    got = out.tolist()
    for i, (k, p) in enumerate(filters):
        mass, edge = kept(x, 0.8, k, p)
        if edge == 0.0 and kind not in ("equal", "two", "halves", "grid"):          # without ties the plain filters keep the same
            assert ((plain_sampling_probs(x.numpy(), 0.8, k, p, 0.0) > 0.0) == (mass > 0.0)).all(), (k, p)
        cdf = np.cumsum(mass) / mass.sum()
        for u, token in zip(us, got[i * len(us):]):
            assert edge > 0.0 or mass[token] > 0.0, (k, p, u)
            # float sums of V terms against float64, and what the edge moves
            slack = 1e-4 + 2 * edge
            assert cdf[token] >= u - slack and (token == 0 or cdf[token - 1] <= u + slack), (k, p, u)


@pytest.mark.parametrize("V", [2000, 20000])          # one block a row; a cluster of blocks
def test_rows_that_are_not_numbers(ops, V):  # noqa: F811
    """An infinite maximum, or a NaN that stays, leaves no sum to draw from: the first largest value is taken.  Top-k drops a NaN:
    what is left is drawn from."""
    x = torch.randn(4, V, generator=torch.Generator().manual_seed(3))
    x[0, 11] = float("nan")
    x[1, 17] = float("inf")
    x[2] = float("nan")
    x[3, 5] = x[3, 1200] = float("inf")
    order = torch.where(x[0].isnan(), -torch.inf, x[0]).argsort(descending=True).tolist()
    f = lambda v, dt=torch.float32: torch.full((4,), v, dtype=dt, device=dev())  # noqa: E731
    for k, p in ((50, 0.9), (50, 1.0), (0, 0.9), (0, 1.0)):
        seen = set()
        for _ in range(3):
            out = torch.empty(4, dtype=torch.int32, device=dev())
            ops.sample(x.to(dev()), f(1.0), f(k, torch.int32), f(p), f(0.0), f(0.4), out)
            got = out.tolist()
            assert got[1:] == [17, 0, 5], (k, p)
            assert got[0] in order[:k or 1], (k, p)
            seen.add(got[0])
        assert len(seen) == 1, (k, p)


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
