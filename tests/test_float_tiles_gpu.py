"""The register-tiled 32-bit kernels (contraction and paged attention) at the edges of their tiles, against float64."""
import pytest
import torch

from tests.test_kernels_gpu import attention_reference, dev, gemm_reference, ops, paged_setup, rnd, tiles_for  # noqa: F401

pytestmark = pytest.mark.gpu

# rows around the heights of 16, 32 and 64; columns around 64 (odd ones too); K from one 16-byte step over ends of a slice
# of 32 to sums that are cut among the blocks of a cluster (few tiles over a long K)
SHAPES = [(4, 66, 36), (5, 66, 36), (9, 64, 4), (16, 63, 28), (17, 65, 32), (32, 2, 36), (33, 129, 100), (64, 128, 896), (65, 66, 4864), (389, 896, 1536),
          # five to eight rows at the edges of what the row-streaming kernel takes of them: slices of K, tiles of features times rows
          (5, 4096, 96), (5, 4097, 96), (8, 64, 64), (8, 64, 68), (8, 64, 256), (9, 64, 256), (8, 64, 260), (7, 9473, 512), (8, 9473, 512), (5, 11361, 512),
          # on the tensor cores: the smallest row counts and work that go there and those beside them, ends of slices of 32 and of
          # tiles of 128 features and 160 tokens, odd features, K cut among 2, 4 and 8 blocks
          (17, 6144, 512), (16, 6144, 512), (32, 6143, 512), (33, 1221, 1024), (33, 1220, 1024), (64, 641, 2052), (160, 896, 896), (161, 8200, 68), (320, 129, 2020),
          (400, 517, 516), (1000, 300, 420), (389, 37889, 36), (389, 896, 4864), (389, 1500, 4)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("epi", [0, 1, 2, 3])
def test_float_contraction(ops, M, N, K, epi):  # noqa: F811
    if epi == 3 and N % 2:
        N += 1
    a, w, bias = rnd((M, K), torch.float32, 1), rnd((N, K), torch.float32, 2, 0.2), rnd((N,), torch.float32, 3)
    residual = rnd((M, N), torch.float32, 4)
    out = None if epi == 2 else torch.full((M, N // 2 if epi == 3 else N), float("nan"), device=dev())
    want = gemm_reference(a, w, bias, epi, residual)
    ops.gemm_simt(a, w, bias, epi, out, residual if epi == 2 else None)
    got = (residual if epi == 2 else out).double().cpu()
    # the rounding of K products and sums, each at most 2^-24 of the sum of magnitudes; a gated pair multiplies two of them
    size = a.abs().double().cpu() @ w.abs().double().cpu().t() + bias.abs().double().cpu() + 4.0
    bound = (K + 4) * 2.0 ** -24 * size
    if epi == 3:
        size, bound = size[:, 0::2] + size[:, 1::2], bound[:, 0::2] + bound[:, 1::2]
        bound = bound * size * 1.2 + 1e-6 * (1.0 + want.abs())
    assert bool(((got - want).abs() <= bound).all())


def on_ffma(ops, a, w):  # noqa: F811
    """The same contraction on CUDA cores: without scratch for the split tokens it stays there."""
    (M, K), N, out = a.shape, w.shape[0], torch.empty((a.shape[0], w.shape[0]), device=dev())
    ops._check(ops.lib().llb_gemm_simt(a.data_ptr(), 0, w.data_ptr(), 0, 0, out.data_ptr(), 0, ops.EPI_STORE, M, N, K, 0, 0,
                                       ops.async_error_flag(dev()).data_ptr(), ops.current_stream()))
    return out


@pytest.mark.parametrize("M,N,K", [s for s in SHAPES if s[0] > 16] + [(389, 9728, 896), (24, 9728, 896), (17, 6200, 4864), (40, 6200, 512), (389, 1500, 8960)])
def test_float_contraction_is_no_further_off_than_ffma(ops, M, N, K):  # noqa: F811
    """The relative 2-norm error against 64 bits, on the tensor cores beside FFMA (which is 1.1 to 3.6 times as far off).  Two parts an
    operand instead of three, a plane in another's place or a product left out are 2.4e-6 and more off at every K, and one accumulation in
    tensor memory over K = 896 8.6e-7."""
    if ops.lib().llb_gemm_simt_scratch_bytes(0, 0, M, N, K) == 0:
        pytest.skip("these sizes stay on CUDA cores")
    a, w, out = rnd((M, K), torch.float32, 11), rnd((N, K), torch.float32, 12), torch.empty((M, N), device=dev())
    ops.gemm_simt(a, w, None, ops.EPI_STORE, out)
    want = a.double() @ w.double().t()
    error, ffma = (float((x.double() - want).norm() / want.norm()) for x in (out, on_ffma(ops, a, w)))
    assert error <= ffma and error < 3e-7, (error, ffma)


# a tile's K in one block, cut among eight and among four; tiles of 96, 48 and 160 tokens, the last feature tile ragged
@pytest.mark.parametrize("M,N,K", [(161, 1030, 516), (40, 128, 10240), (320, 1299, 2020)])
def test_float_contraction_of_what_bf16_does_not_hold(ops, M, N, K):  # noqa: F811
    """Infinities, NaN, values that round to infinity in bf16 and sums beyond the floats, among ordinary rows, on the tensor cores."""
    assert ops.lib().llb_gemm_simt_scratch_bytes(0, 0, M, N, K) > 0
    a, w = rnd((M, K), torch.float32, 1), rnd((N, K), torch.float32, 2, 0.2)
    w = torch.where(w.abs() < 1e-3, torch.full_like(w, 1e-3), w)          # (no zero: infinity times it is NaN)
    a[0, K // 2], a[1, 3], a[2, K - 1], a[3, :2] = float("inf"), -float("inf"), float("nan"), float("inf")
    a[4], a[4, 5], a[5, 7], a[6] = 0.0, 3.4e38, -3.39e38, 3.3e38
    a[7] *= 1e-37
    w[9, 0], w[9, 1] = 1.0, -1.0          # row 3 meets infinity minus infinity there
    out = torch.full((M, N), 7.0, device=dev())
    ops.gemm_simt(a, w, None, ops.EPI_STORE, out)
    want, got = (a.double() @ w.double().t()).cpu(), out.double().cpu()
    size = (a.abs().double() @ w.abs().double().t()).cpu()
    bound = (K + 4) * 2.0 ** -24 * size
    safe = torch.isfinite(want) & (size < 3.0e38)                  # (no order of the sum passes the largest float)
    assert bool(((got - want).abs()[safe] <= bound[safe]).all()) and int(safe.sum()) >= (M - 6) * N
    assert bool((got[:2] == want[:2]).all()) and bool(torch.isnan(got[2]).all()) and bool(torch.isnan(got[3, 9]))
    same_sign = (w[:, 0] * w[:, 1] > 0).cpu()
    assert bool((got[3][same_sign] == want[3][same_sign]).all())
    beyond = torch.isfinite(want[6]) & (want[6].abs() < 3.0e38) | torch.isnan(got[6]) | torch.isinf(got[6])
    assert bool(beyond.all())          # sums that pass the largest float on the way are infinite or NaN, as with FFMA


def test_a_nan_does_not_make_a_float_contraction_slow(ops):  # noqa: F811
    """The tiles whose sums are no finite number are done again in float arithmetic: 7 times the time of finite ones here, where FFMA
    throughout is 4 (every thread from memory by itself: 450)."""
    a, w, out = rnd((389, 896), torch.float32, 23), rnd((9728, 896), torch.float32, 24, 0.02), torch.empty((389, 9728), device=dev())

    def best():
        times = []
        for _ in range(5):
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            begin.record()
            for _ in range(4):
                ops.gemm_simt(a, w, None, ops.EPI_STORE, out)
            end.record()
            end.synchronize()
            times.append(begin.elapsed_time(end))
        return min(times)
    finite = best()
    a[:, 5] = float("nan")
    assert best() < 10 * finite and bool(torch.isnan(out).all())


@pytest.mark.parametrize("M,N,K", [(161, 1030, 516), (40, 128, 10240)])
@pytest.mark.parametrize("small", [1e-32, 1e-34, 1e-36, 1e-38, 1e-40])
@pytest.mark.parametrize("which", ["tokens", "weights"])
def test_float_contraction_of_numbers_below_what_three_bf16_hold(ops, M, N, K, small, which):  # noqa: F811
    """Operands down to the subnormal floats keep all the bits that they have; the other operand is large, so that the sums are ordinary."""
    assert ops.lib().llb_gemm_simt_scratch_bytes(0, 0, M, N, K) > 0
    a, w = rnd((M, K), torch.float32, 21), rnd((N, K), torch.float32, 22)
    if which == "tokens":
        a, w = (a.double() * small).float(), w * 1e9
    else:
        a, w = a * 1e9, (w.double() * small).float()
    out = torch.full((M, N), float("nan"), device=dev())
    ops.gemm_simt(a, w, None, ops.EPI_STORE, out)
    want = a.double() @ w.double().t()
    # as for ordinary numbers: 1.4e-7 at the longest K (FFMA 2.7e-7 to 4e-7)
    assert float((out.double() - want).norm() / want.norm()) < 3e-7


@pytest.mark.parametrize("Hq,Hkv,hd", [(14, 2, 64), (3, 3, 128), (12, 2, 128)])
@pytest.mark.parametrize("window", [None, 70])
@pytest.mark.parametrize("groups", [2, 4])
def test_float_attention_by_groups(ops, Hq, Hkv, hd, window, groups):  # noqa: F811
    """Groups of warps that share a block's keys: fewer tiles of keys than groups, as many, and more; windows that leave groups without."""
    lens, starts = [1, 16, 67, 33, 20], [0, 63, 0, 130, 440]
    s = paged_setup(torch.float32, lens, starts, Hq, Hkv, hd, 16, 13)
    ts, tq, nt = tiles_for(lens, 16)
    outs = []
    for nsplit in (1, -groups):
        out = torch.full((s["rows"], Hq * hd), float("nan"), device=dev())
        ops.paged_attention_simt(s["q"], s["kc"], s["vc"], out, ts, tq, nt, s["span_row"], s["span_len"], s["span_pos"], s["bt"],
                                 s["max_pages"], 16, Hq, Hkv, hd, window or 0, hd ** -0.5, 16, nsplit)
        outs.append(out.cpu())
    ref = attention_reference(s["full"], lens, starts, hd, window).reshape(s["rows"], Hq * hd)
    assert not torch.isnan(outs[1]).any()
    assert torch.allclose(outs[1], ref, atol=2e-5, rtol=2e-5) and torch.allclose(outs[0], outs[1], atol=2e-6, rtol=2e-6)


@pytest.mark.parametrize("Hq,Hkv,hd", [(14, 2, 64), (3, 3, 128), (9, 1, 64), (12, 2, 128)])
@pytest.mark.parametrize("window", [None, 33])
@pytest.mark.parametrize("bq", [16, 5])
def test_float_attention(ops, Hq, Hkv, hd, window, bq):  # noqa: F811
    lens, starts = [1, 16, 67, 33], [0, 63, 0, 130]
    s = paged_setup(torch.float32, lens, starts, Hq, Hkv, hd, 16, 11)
    ts, tq, nt = tiles_for(lens, bq)
    out = torch.full((s["rows"], Hq * hd), float("nan"), device=dev())
    ops.paged_attention_simt(s["q"], s["kc"], s["vc"], out, ts, tq, nt, s["span_row"], s["span_len"], s["span_pos"], s["bt"],
                             s["max_pages"], 16, Hq, Hkv, hd, window or 0, hd ** -0.5, bq)
    ref = attention_reference(s["full"], lens, starts, hd, window).reshape(s["rows"], Hq * hd)
    got = out.cpu()
    assert not torch.isnan(got).any()
    assert torch.allclose(got, ref, atol=2e-5, rtol=2e-5), f"max diff {float((got - ref).abs().max())}"


@pytest.mark.parametrize("Hq,Hkv,hd", [(6, 2, 64), (6, 2, 128), (4, 4, 128), (9, 1, 128)])
@pytest.mark.parametrize("window,keep", [(0, 0), (33, 5), (70, 66), (-24, 0)])
def test_float_attention_with_all_that_scores_take(ops, Hq, Hkv, hd, window, keep):  # noqa: F811
    """Cap, slopes, sinks, a window (or a block of positions) and first keys that stay, against float64."""
    lens, starts, cap, bq = [1, 16, 67, 33], [0, 63, 0, 130], 6.0, 16
    s = paged_setup(torch.float32, lens, starts, Hq, Hkv, hd, 16, 12)
    sinks, slopes = rnd((Hq,), torch.float32, 5), rnd((Hq,), torch.float32, 6, 0.05).abs()
    ts, tq, nt = tiles_for(lens, bq)
    out = torch.full((s["rows"], Hq * hd), float("nan"), device=dev())
    ops.paged_attention_simt(s["q"], s["kc"], s["vc"], out, ts, tq, nt, s["span_row"], s["span_len"], s["span_pos"], s["bt"],
                             s["max_pages"], 16, Hq, Hkv, hd, window, hd ** -0.5, bq, sinks=sinks, softcap=cap, keep=keep, slopes=slopes)
    want = []
    for (q, k, v), n, start in zip(s["full"], lens, starts):
        q, k, v = q.double()[start:], k.double().repeat_interleave(Hq // Hkv, 1), v.double().repeat_interleave(Hq // Hkv, 1)
        at, key = torch.arange(start, start + n)[:, None], torch.arange(start + n)[None]
        first = at - window + 1 if window > 0 else at - at % -window if window < 0 else torch.zeros_like(at)
        visible = (key <= at) & ((key >= first) | (key < keep))
        x = cap * torch.tanh(torch.einsum("qhd,khd->hqk", q, k) * hd ** -0.5 / cap)
        x = x - slopes.double().cpu()[:, None, None] * (at - key)
        e = torch.where(visible, x.exp(), 0.0)          # (scores are at most the cap: no maximum to take off)
        den = e.sum(-1) + sinks.double().cpu()[:, None].exp()
        want.append(torch.einsum("hqk,khd->qhd", e / den[:, :, None], v).reshape(n, Hq * hd))
    want, got = torch.cat(want), out.double().cpu()
    assert not torch.isnan(got).any()
    assert torch.allclose(got, want, atol=2e-5, rtol=2e-5), f"max diff {float((got - want).abs().max())}"


def test_a_tile_too_high_is_refused(ops):  # noqa: F811
    """A tile whose rows the general kernel's shared memory cannot hold is refused in every dtype, at any address."""
    from lightllm_b200.csrc.ops import KernelError
    s = paged_setup(torch.float32, [500], [0], 2, 2, 64, 16, 3)
    ts, tq, nt = tiles_for([500], 500)
    out = torch.empty((500, 128), device=dev())
    with pytest.raises(KernelError, match="use a smaller BQ"):
        ops.paged_attention_simt(s["q"], s["kc"], s["vc"], out, ts, tq, nt, s["span_row"], s["span_len"], s["span_pos"], s["bt"],
                                 s["max_pages"], 16, 2, 2, 64, 0, 0.125, 500)


def test_too_many_rows_are_refused(ops):  # noqa: F811
    """One row more than 65,535 tiles of 64 hold is refused whether or not the operands' rows are 16-byte steps."""
    from lightllm_b200.csrc.ops import KernelError
    for K in (4, 5):
        a, w = torch.zeros((65535 * 64 + 1, K), device=dev()), torch.zeros((4, K), device=dev())
        with pytest.raises(KernelError, match="too large for one launch"):
            ops.gemm_simt(a, w, None, 0, torch.empty((a.shape[0], 4), device=dev()))
