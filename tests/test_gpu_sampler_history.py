"""The sampler's repetition penalty for histories that crowd one block of logits, repeat a token, fill the device's history or hold ids outside
the vocabulary: the count of a token decides how often the penalty is applied, in the exact-order kernel and in the tree sampler."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def history_of(kind, V, rng):
    n = {"full": 4096}.get(kind, 300)
    if kind == "one":
        return np.full(n, V - 1, np.int32)
    if kind == "crowded":  # one block of 2048 logits, across a multiple of the block's threads
        return rng.integers(500, 530, n).astype(np.int32)
    h = rng.integers(0, V, n).astype(np.int32)
    if kind == "outside":
        h[::3], h[1::3] = V, -1
    return h


@pytest.mark.parametrize("V", [320, 2049, 128256, 400000])  # the last one is the tree sampler's
@pytest.mark.parametrize("kind", ["one", "crowded", "outside", "full"])
def test_penalty_counts(oracle, V, kind):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from lighterpp_b200 import ops
    rng = np.random.default_rng([V, len(kind)])
    hist = history_of(kind, V, rng)
    if V < 531 and kind == "crowded":
        hist %= V
    out = torch.zeros(1, dtype=torch.int32, device="cuda")
    lg = rng.standard_normal(V).astype(np.float32)
    inside = hist[(hist >= 0) & (hist < V)]
    lg[inside] += np.float32(3.0)  # the penalised ones lead, so that one application too few or too many shows in the order
    times = np.bincount(inside, minlength=V)
    want = lg.copy()
    for t in np.flatnonzero(times):  # the penalty in FP32, once per occurrence, as the kernel and the reference do
        for _ in range(times[t]):
            want[t] = want[t] / np.float32(1.01) if want[t] > 0 else want[t] * np.float32(1.01)
    for temperature, r in ((0.0, 0.0), (0.8, 0.3), (0.8, 0.9)):
        if V == 400000 and temperature:
            continue  # its categorical sums are re-associated
        d = torch.from_numpy(lg).cuda()
        ops.cuda_sample(d, V, temperature, 1.01, torch.from_numpy(hist).cuda(), len(hist), r, out)
        assert int(out.item()) == (int(want.argmax()) if not temperature else oracle.sample_twin(want, temperature, 1.0, np.zeros(0, np.int32), r))
