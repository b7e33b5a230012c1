"""The stand-alone operators at the sizes where their kernels change over: parts of a row shared by several warps, remainders of a
batch of loads, positions that do not fill a cluster, head sizes and addresses that the vector kernels do not take.  Against
64-bit sums; the bound of a sum of n products is n + 8 roundings of the sum of magnitudes, 2^-24 each."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def T():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return torch


def close(got, ref, magnitudes, n):
    assert got.shape == ref.shape
    assert np.all(np.abs(got.astype(np.float64) - ref) <= (n + 8) * 2.0 ** -24 * magnitudes + 1e-30)


@pytest.mark.parametrize("n,d,dt,shift", [(1, 8, "f16", 0), (3, 8, "f16", 0), (5, 1032, "f16", 0), (17, 2048, "f16", 0), (1024, 4096, "f16", 0),
                                          (593, 5632, "f16", 0), (4737, 288, "f16", 0), (9473, 1016, "f16", 0), (31, 51200, "f16", 0),
                                          (64, 51208, "f16", 0), (100, 4096, "f16", 1), (7, 12, "f32", 0), (288, 768, "f32", 0),
                                          (4800, 772, "f32", 0), (12, 2048, "f32", 1)])
def test_gemv(T, n, d, dt, shift):
    from lighterpp_b200 import ops
    g = T.Generator(device="cuda").manual_seed(n * 7 + d)
    wide = T.randn(n * d + shift, device="cuda", generator=g, dtype=T.float16 if dt == "f16" else T.float32)
    w = wide[shift:].view(n, d)  # shift = 1: rows off the 16-byte boundary
    x = T.randn(d, device="cuda", generator=g)
    out = T.full((n + 1,), 7.0, device="cuda")
    ops.cuda_gemv(out, x, w, n, d, ops.WEIGHT_FP16 if dt == "f16" else ops.WEIGHT_FP32)
    W, X = w.double(), x.double()
    close(out[:n].cpu().numpy(), (W @ X).cpu().numpy(), (W.abs() @ X.abs()).cpu().numpy(), d)
    assert out[n].item() == 7.0


@pytest.mark.parametrize("n", [1, 31, 1024, 1025, 8192, 8193, 20000])
def test_rmsnorm(T, n):
    from lighterpp_b200 import ops
    g = T.Generator(device="cuda").manual_seed(n)
    x, w = T.randn(n, device="cuda", generator=g), T.randn(n, device="cuda", generator=g)
    out = T.empty_like(x)
    ops.cuda_rmsnorm(out, x, w, n)
    X = x.double()
    ref = X / T.sqrt((X * X).mean() + 1e-5) * w.double()
    # the mean of squares is a sum of positive terms: half of its n / 1024 + 16 roundings, and four of the factors
    assert ((out.double() - ref).abs() <= (n / 1024 + 32) * 2.0 ** -24 * ref.abs() + 1e-30).all()


@pytest.mark.parametrize("positions", [1, 7, 8, 9, 127, 128, 129, 1501])
@pytest.mark.parametrize("hs,gqa,shift", [(8, 1, 0), (16, 2, 0), (48, 1, 0), (64, 4, 0), (96, 3, 0), (128, 4, 0), (128, 1, 1), (36, 2, 0)])
def test_scores_and_aggregation(T, positions, hs, gqa, shift):
    from lighterpp_b200 import ops
    kvh, rows, layer = 3, positions + 5, 1
    heads = kvh * gqa
    g = T.Generator(device="cuda").manual_seed(positions * 1000 + hs)
    # rows beyond the positions hold NaN: they must not be touched
    wide = T.randn(2 * kvh * rows * hs + shift, device="cuda", generator=g, dtype=T.float16)
    cache = wide[shift:].view(2, kvh, rows, hs)
    cache[:, :, positions:] = float("nan")
    q = T.randn((heads, hs), device="cuda", generator=g)
    att = T.full((heads, rows), 7.0, device="cuda")
    ops.cuda_multihead_gemv(att, q, cache, layer, positions - 1, heads, kvh, hs, rows)
    K, Q = cache[layer, :, :positions].double().repeat_interleave(gqa, 0), q.double()
    close(att[:, :positions].cpu().numpy(), T.einsum("hd,htd->ht", Q, K).cpu().numpy(), T.einsum("hd,htd->ht", Q.abs(), K.abs()).cpu().numpy(), hs)
    assert (att[:, positions:] == 7.0).all()
    p = T.rand((heads, rows), device="cuda", generator=g)
    out = T.full((heads * hs + 1,), 7.0, device="cuda")
    ops.cuda_aggregation_multihead(out, cache[layer], p, heads, positions, hs, gqa, rows)
    P = p[:, :positions].double()
    close(out[:-1].view(heads, hs).cpu().numpy(), T.einsum("ht,htd->hd", P, K).cpu().numpy(), T.einsum("ht,htd->hd", P, K.abs()).cpu().numpy(), positions)
    assert out[-1].item() == 7.0


def test_operators_captured_in_a_graph(T):
    """A stream that is being captured, with a copy before the first operator."""
    from lighterpp_b200 import ops
    n = 512
    x, w = T.randn(n, device="cuda"), T.randn((n, n), device="cuda", dtype=T.float16)
    a, b, src = T.empty(n, device="cuda"), T.empty(n, device="cuda"), T.randn(n, device="cuda")
    ones = T.ones(n, device="cuda")
    stream = T.cuda.Stream()
    graph = T.cuda.CUDAGraph()
    with T.cuda.graph(graph, stream=stream):
        x.copy_(src)
        ops.cuda_rmsnorm(a, x, ones, n)
        ops.cuda_gemv(b, a, w, n, n, ops.WEIGHT_FP16)
        ops.cuda_residual_add(a, a, b, n)
    for k in range(2):
        src.normal_()
        graph.replay()
        T.cuda.synchronize()
        X = src.double()
        h = X / T.sqrt((X * X).mean() + 1e-5)
        ref = h + w.double() @ h
        assert (a.double() - ref).abs().max() <= 600 * 2.0 ** -24 * (w.double().abs() @ h.abs()).max()


@pytest.mark.parametrize("positions", [1, 2, 7, 9])
def test_aggregation_of_few_positions_in_a_graph(T, positions):
    """Most CTAs of a cluster have no position and go straight to handing over their (empty) sums, 64 launches one behind the other."""
    from lighterpp_b200 import ops
    heads, hs, rows = 32, 128, 16
    v = T.randn((heads, rows, hs), device="cuda", dtype=T.float16)
    att, out = T.rand((64, heads, rows), device="cuda"), T.zeros((64, heads * hs), device="cuda")
    graph = T.cuda.CUDAGraph()
    with T.cuda.graph(graph):
        for k in range(64):
            ops.cuda_aggregation_multihead(out[k], v, att[k], heads, positions, hs, 1, rows)
    for _ in range(3):
        att.uniform_()
        out.zero_()
        graph.replay()
        P, V = att[:, :, :positions].double(), v[:, :positions].double()
        close(out.view(64, heads, hs).cpu().numpy(), T.einsum("kht,htd->khd", P, V).cpu().numpy(), T.einsum("kht,htd->khd", P, V.abs()).cpu().numpy(), positions)
