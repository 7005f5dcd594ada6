"""Decode attention where it reads keys before the kernel before it has completed, and where all requests' keys are cut together."""
import math
import random

import pytest
import torch

from lightllm_b200 import EngineCore, EngineOptions, StepEntry, write_random_model
from tests.plain import qwen2_plain as P
from tests.test_kernels_gpu import dev, ops, paged_setup, rnd, tiles_for  # noqa: F401
from tests.tiny_configs import config
from tests.tolerances import atol_for

pytestmark = pytest.mark.gpu


def plain_rows(full, starts, hd, window=0, keep=0, softcap=0.0, slopes=None, sinks=None, cross=1):
    """Each request's last query against its keys, in 64 bits: [requests, Hq, cross, hd]."""
    out = []
    for (q, k, v), s in zip(full, starts):
        q, k, v = q[s].double(), k[: s + 1].double(), v[: s + 1].double()
        Hq, Hkv, pos = q.shape[0], k.shape[1], torch.arange(s + 1)
        first = max(0, s - window + 1) if window > 0 else s - s % -window if window < 0 else 0
        sc = torch.einsum("hd,phd->hp", q, k.repeat_interleave(Hq // Hkv, 1)) * hd ** -0.5
        if softcap:
            sc = softcap * torch.tanh(sc / softcap)
        if slopes is not None:
            sc = sc - slopes.double().cpu()[:, None] * (s - pos)
        sc = sc.masked_fill(~((pos >= first) | (pos < keep)), -math.inf)
        p = torch.exp(sc - sc.max(-1, keepdim=True).values)
        den = p.sum(-1) + (torch.exp(sinks.double().cpu() - sc.max(-1).values) if sinks is not None else 0.0)
        p = p / den[:, None]
        if cross > 1:
            out.append(torch.einsum("hp,pgd->hgd", p, v))
        else:
            out.append(torch.einsum("hp,phd->hd", p, v.repeat_interleave(Hq // Hkv, 1))[:, None])
    return torch.stack(out)


OPTIONS = [dict(), dict(sinks=True), dict(softcap=20.0), dict(slopes=True), dict(window=100, keep=5), dict(window=-96, keep=3), dict(window=-96),
           dict(cross=True), dict(cross=True, slopes=True, window=70, keep=70), dict(out_float=True),
           dict(sinks=True, softcap=15.0, slopes=True, window=200, keep=17, out_float=True)]
# ends of tiles of 16 and 32 keys, of a round of four warps' tiles, and one key and 64 keys off them
STARTS = [0, 14, 15, 16, 31, 32, 33, 63, 64, 95, 96, 127, 128, 129, 191, 192, 700, 2000]


@pytest.mark.parametrize("option", OPTIONS, ids=lambda o: "-".join(o) or "plain")
@pytest.mark.parametrize("Hq,Hkv,hd", [(14, 2, 64), (12, 2, 128)])
@pytest.mark.parametrize("nsplit", [1, 6, -18, -40, -150])
def test_everything_that_scores_take(ops, option, Hq, Hkv, hd, nsplit):  # noqa: F811
    """Requests cut one by one (in a cluster) and together (pieces of one length), with every option that either shares its code with."""
    s = paged_setup(torch.bfloat16, [1] * len(STARTS), STARTS, Hq, Hkv, hd, 16, seed=91)
    ts, tq, nt = tiles_for([1] * len(STARTS), 1)
    cross = Hkv if option.get("cross") else 1
    slopes = 2.0 ** (-1.0 - torch.arange(Hq) % 8).float().to(dev()) if option.get("slopes") else None
    sinks = rnd((Hq,), torch.float32, 92, 2.0) if option.get("sinks") else None
    kw = dict(window=option.get("window", 0), keep=option.get("keep", 0), softcap=option.get("softcap", 0.0))
    want = plain_rows(s["full"], STARTS, hd, slopes=slopes, sinks=sinks, cross=cross, **kw).reshape(nt, -1)
    for fresh in (0, 1, 64):
        out = torch.full((nt, Hq * cross * hd), float("nan"), dtype=torch.float32 if option.get("out_float") else torch.bfloat16, device=dev())
        scratch = torch.full((max(1, -nsplit) * Hq * cross * (hd + 2),), float("nan"), device=dev())
        ops.paged_decode_mma(s["q"], s["kc"], s["vc"], out, ts, tq, nt, s["span_row"], s["span_pos"], s["bt"], s["max_pages"], 16, Hq, Hkv,
                             hd, kw["window"], hd ** -0.5, nsplit, scratch, sinks=sinks, cross=cross, softcap=kw["softcap"], keep=kw["keep"],
                             slopes=slopes, fresh=fresh)
        got = out.double().cpu()
        assert not torch.isnan(got).any()
        # probabilities are bf16 operands (2^-9 of a value each, values of up to 4.5) and so is the result
        assert torch.allclose(got, want, atol=2e-2, rtol=2e-2), f"max diff {float((got - want).abs().max())}"


@pytest.mark.parametrize("Hq,Hkv,hd", [(14, 2, 64), (12, 2, 128)])
@pytest.mark.parametrize("rows", ["requests", 0, 33, 500, 2000])
@pytest.mark.parametrize("nsplit", [1, 5, 8, -64, -130])
def test_keys_that_the_kernel_before_writes(ops, Hq, Hkv, hd, rows, nsplit):  # noqa: F811
    """The projection writes the newest keys and values and the attention follows it without a wait on the host: one token of each of
    64 requests, or 64 tokens of one request from a position on, each a row of its own.  The places are poisoned before every
    pass, so a key read too early shows; the result is that of the same launches with a wait between them, bit by bit."""
    M, K, page = 64, 256, 16
    if rows == "requests":
        starts, fresh = [(37 * i * i) % 1400 for i in range(M - len(STARTS))] + STARTS, 1
        spans = [(i, s) for i, s in enumerate(starts)]
    else:
        fresh, spans = 64, [(0, rows + i) for i in range(M)]
    longest = [max(s for r, s in spans if r == i) for i in range(max(r for r, _ in spans) + 1)]
    pages = -(-(max(longest) + 1) // page)
    kc, vc = (rnd((len(longest) * pages * page, Hkv, hd), torch.bfloat16, 93 + i) for i in range(2))
    order = torch.randperm(len(longest) * pages, generator=torch.Generator().manual_seed(95)).reshape(len(longest), pages)
    bt = order[torch.tensor([r for r, _ in spans])].to(torch.int32).to(dev())
    pos = torch.tensor([s for _, s in spans], dtype=torch.int32, device=dev())
    slots = torch.tensor([int(order[r, s // page]) * page + s % page for r, s in spans], dtype=torch.int32, device=dev())
    N = (Hq + 2 * Hkv) * hd
    w, a, x = rnd((N, K), torch.bfloat16, 96, 0.1), rnd((M, K), torch.bfloat16, 97), rnd((M, K), torch.float32, 98)
    one, normed = torch.ones(K, device=dev()), torch.empty((M, K), dtype=torch.bfloat16, device=dev())
    inv = (10000.0 ** (-torch.arange(0, hd, 2, dtype=torch.float64) / hd)).float().to(dev())
    table, iota, zeros = ops.rope_table(pos, inv), torch.arange(M, dtype=torch.int32, device=dev()), torch.zeros(M, dtype=torch.int32, device=dev())
    q, out = (torch.empty((M, Hq * hd), dtype=torch.bfloat16, device=dev()) for _ in range(2))
    scratch = torch.empty(max(1, -nsplit) * Hq * (hd + 2), device=dev())

    def run(fresh, wait):
        kc[slots.long()], vc[slots.long()] = float("nan"), float("nan")
        out.fill_(float("nan"))
        torch.cuda.synchronize()
        ops.rmsnorm(x, one, 1e-6, normed)          # (gives its early word before its own wait)
        ops.gemm_decode(w, ops.DEPI_ROPE_KV, M, a=a, slot_mapping=slots, split_k=0, rope_table=table, rotary_dim=hd, num_heads=Hq,
                        num_kv_heads=Hkv, head_dim=hd, q_out=q, k_cache=kc, v_cache=vc)
        if wait:
            torch.cuda.synchronize()
        ops.paged_decode_mma(q, kc, vc, out, iota, zeros, M, iota, pos, bt, pages, page, Hq, Hkv, hd, 0, hd ** -0.5, nsplit, scratch, fresh=fresh)
        return out.clone()

    want = run(0, True)
    assert not torch.isnan(want).any()
    for _ in range(5):
        assert torch.equal(run(fresh, False), want)
    ops.check_async_errors(dev())


@pytest.mark.parametrize("native", ["1", "0"])
@pytest.mark.parametrize("rowwise", ["1", "0"])
def test_requests_of_very_different_lengths(tmp_path, monkeypatch, native, rowwise):
    """Batches whose longest request is far longer than the rest (their keys are cut together), alone and beside a portion, launched one
    by one and from a graph, follow the plain implementation."""
    monkeypatch.setenv("LLB_NATIVE_STEP", native)
    monkeypatch.setenv("LLB_ROWWISE_STEPS", rowwise)
    monkeypatch.setenv("LLB_FUSED_DECODE", "0")
    d, cfg = str(tmp_path / "model"), dict(config("E"), max_position_embeddings=4096)
    write_random_model(cfg, 61, d, "bfloat16")
    cfg, w = P.read_model_dir(d)
    rng = random.Random(62)
    held = [2500, 40, 9, 300]
    seqs = [[rng.randrange(cfg["vocab_size"]) for _ in range(n + 20)] for n in held]
    ref = {i: P.plain_forward(cfg, w, s) for i, s in enumerate(seqs)}
    core = EngineCore(d, EngineOptions(dtype="bfloat16", max_seq_len=4096, max_batch_tokens=4096, page_size=16, num_pages=220, max_seqs=8))
    at, worst, cut = list(held), 0.0, 0
    for i in range(4):
        core.open(i)
    core.step([StepEntry(i, seqs[i][:n], []) for i, n in enumerate(held)])

    def step(parts):
        nonlocal worst, cut
        out = core.step([StepEntry(i, seqs[i][at[i]: at[i] + n], [n - 1]) for i, n in parts])
        cut += any(k[0] == "even" for k in core.runner.last_ctx.shape_key if isinstance(k, tuple))
        for k, (i, n) in enumerate(parts):
            at[i] += n
            worst = max(worst, float((out[k].float().cpu() - ref[i][at[i] - 1]).abs().max()))

    for _ in range(5):
        step([(0, 1), (1, 1), (2, 1), (3, 1)])
    for _ in range(2):
        step([(0, 1), (1, 1), (2, 3), (3, 1)])
    core.runner.check_device_errors()
    assert cut >= 6 and core.runner.graph_replays > 0
    assert worst <= atol_for("E", "bfloat16", ref), worst
