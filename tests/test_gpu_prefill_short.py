"""Prompt blocks of at most 64 tokens, whose activation tiles have 16, 32, 48 or 64 rows, against the token loop: token counts around
every tile, feed-forward widths with a ragged last row tile and of more tiles than SMs, wanted logits of one and of all tokens,
grouped weights (per-head matrices), BF16 and FP16."""
import numpy as np
import pytest

from lighterpp_b200 import synth
from lighterpp_b200.formats import ModelConfig

pytestmark = pytest.mark.gpu
SIZES = (2, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64)


@pytest.fixture(scope="module")
def E():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from lighterpp_b200 import engine
    return engine


def compare(batched, loop, toks, bound):
    ref = loop.extend(toks[:64], 0, range(64))

    def check(got, rows):
        err = np.linalg.norm(got - ref[rows], axis=1) / np.linalg.norm(ref[rows], axis=1)
        assert np.isfinite(got).all() and err.max() <= bound, (err.max(), rows[int(err.argmax())])

    for n in SIZES:
        check(batched.extend(toks[:n], 0, range(n)), list(range(n)))
    for n in (16, 33):  # behind a cache, the last token's logits only
        batched.extend(toks[:30], 0)
        check(batched.extend(toks[30:30 + n], 30, [n - 1]), [29 + n])


# 2 x ff rows: 1408 (11 row tiles) and 1472 (a ragged twelfth), 18944 and 19072 (148 and 149: one and two rounds of the SMs)
@pytest.mark.parametrize("ff", [704, 736, 9472, 9536])
def test_llama(E, ff):
    c = ModelConfig(256, ff, 2, 4, 2, 1000, 96, 10000.0)
    T = synth.gen_model(c, 9, "f16", True)
    engines = [E.Engine(c, "f16", "f16", flags=f) for f in (0, E.FLAG_NO_PREFILL_GEMM)]
    for e in engines:
        e.load_weights(T)
    compare(*engines, synth.prompt_tokens(c.vocab_size, 64, 9), 2e-3)  # FP16 cache rows, queries and probabilities: 2^-11 each
    for e in engines:
        e.close()


def test_latent(E):
    from lighterpp_b200.models import ARCHITECTURES
    from oracle import rutenex
    rot = {"base": 1e4, "dims": 16, "scaling": {"factor": 4.0, "original": 64, "fast": 8.0, "slow": 1.0}}
    mix = {"heads": 5, "dim": 40, "rot_dim": 16, "vdim": 24, "kv_rank": 72, "scale": 56 ** -0.5, "mask": {"size": 20}, "rot": rot}
    cfg = {"architecture": "Rutenex", "width": 136, "vocab": 320, "norm": {"eps": 1e-5},
           "layers": [{"type": "latent_attention", "mixer": mix, "mlp": {"kind": "dense", "ff": 200}}] * 2}
    W, arch = rutenex.random_weights(cfg, 3), ARCHITECTURES["Rutenex"]
    c = arch.configure(cfg, 96)
    engines = [E.Engine(c, "bf16", "f16", flags=f) for f in (0, E.FLAG_NO_PREFILL_GEMM)]
    for e in engines:
        for ours, layer, name, _ in arch.tensors(c):
            e.upload(ours, (np.ascontiguousarray(W[name], dtype=np.float32).view(np.uint32) >> 16).astype(np.uint16), layer)
        e.finalize()
    compare(*engines, np.random.default_rng(4).integers(0, cfg["vocab"], 64), 4e-3)  # the bound of these models' other tests
    for e in engines:
        e.close()
