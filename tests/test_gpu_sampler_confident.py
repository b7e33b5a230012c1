"""The exact-order sampler on distributions whose running sum stays near a power of two (confident ones), holds masked
tokens, or is far below the maximum for most of the vocabulary: ids equal those of the CPU twin on every draw."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engines():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from lighterpp_b200 import engine as E, synth
    out = {}
    for name in ("tiny-f32", "vocab32k-f16", "vocab50k-f16", "vocab128k-f16"):
        c, dt, tied, seed, T = synth.named(name)
        out[c.vocab_size] = E.Engine(c, dt, "f16" if dt == "f16" else "f32")
        out[c.vocab_size].load_weights(T)
    yield out
    for e in out.values():
        e.close()


def logits_of(kind, V, rng):
    lg = rng.standard_normal(V).astype(np.float32)
    at = {"first": 0, "last": V - 1}.get(kind.split("-")[-1], int(rng.integers(1, V - 1)))
    rest = np.log(np.exp(lg.astype(np.float64)).sum())
    if kind.startswith("peak"):  # probability 1 - 10^-k on one token
        lg[at] = rest + float(kind.split("-")[1]) * np.log(10.0)
    elif kind.startswith("two"):  # the sum passes 1 in the middle and stays just above it
        lg[at] = lg[V // 3] = rest + 9.0
    elif kind == "flat-below":  # every other token below half an ulp of the peak
        lg[:], lg[at] = -20.0, 0.0
    elif kind == "masked":
        lg[rng.random(V) < 0.97] = -np.inf
    elif kind == "lowest":
        lg[rng.random(V) < 0.97] = np.finfo(np.float32).min
    elif kind == "one-left":
        lg[:], lg[at] = -np.inf, 1.0
    elif kind == "far":  # a peak so high that the rest is subnormal or zero
        lg[at] = 95.0
    elif kind == "farther":
        lg[at] = 300.0
    elif kind == "nan":
        lg[at] = np.nan
    return lg


KINDS = ["peak-2-first", "peak-2-mid", "peak-3-mid", "peak-4-first", "peak-4-mid", "peak-4-last", "peak-6-mid", "peak-8-first", "two-mid",
         "flat-below", "masked", "lowest", "one-left", "far", "farther", "nan"]


@pytest.mark.parametrize("V", [320, 32000, 50264, 128256])
@pytest.mark.parametrize("kind", KINDS)
def test_ids_equal_the_twin(engines, oracle, V, kind):
    rng = np.random.default_rng([V, KINDS.index(kind)])
    eng = engines[V]
    for s in range(2):
        lg = logits_of(kind, V, rng)
        hist = rng.integers(0, V, size=(0, 64)[s]).astype(np.int32)
        one = np.float32(1.0)
        rs = np.concatenate([rng.random(6), 1 - 10.0 ** -rng.uniform(1, 7, 6), 10.0 ** -rng.uniform(1, 7, 3), [0.0, one, one - np.float32(2 ** -24)]])
        for r in rs.astype(np.float32):
            assert eng.sample(lg, (1.0, 0.8)[s], (1.0, 1.1)[s], hist, float(r)) == oracle.sample_twin(lg, (1.0, 0.8)[s], (1.0, 1.1)[s], hist, float(r)), \
                (s, float(r))
