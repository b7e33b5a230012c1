"""Attention over shared rows of prompt blocks with enough row tiles for the tcgen05 kernel, against the token loop: one and two
CTAs per row tile, heads that do and do not divide 128 rows, rows that are no multiple of 64 columns, windows that begin
inside a tile of keys, none at all, groups, score caps, gates, token counts around the row tiles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def E():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from lighterpp_b200 import engine
    return engine


ROT = {"base": 1e4, "dims": 16, "scaling": {"factor": 4.0, "original": 64, "fast": 8.0, "slow": 1.0}}


def latent(heads, rank, rot_dim, window):
    m = {"heads": heads, "dim": 24, "rot_dim": rot_dim, "vdim": 24, "kv_rank": rank, "scale": 40 ** -0.5, "rot": dict(ROT, dims=rot_dim)}
    if window:
        m["mask"] = {"size": window}
    return {"architecture": "Rutenex", "width": 136, "vocab": 320, "norm": {"eps": 1e-5},
            "layers": [{"type": "latent_attention", "mixer": m, "mlp": None}] * 2}


def shared(heads, kv, dim, window, cap):
    m = {"heads": heads, "kv_heads": kv, "dim": dim, "vdim": dim, "scale": 2.0 * dim ** -0.5, "rot": ROT}
    if window:
        m["mask"] = {"size": window}
    if cap:
        m["softcap"] = cap
    return {"architecture": "Kolatar", "width": 112, "vocab": 300, "norm": {"eps": 1e-5}, "embedding": {"scale": 10.0}, "logit_scale": 1.5, "loop": {"start": 0, "stop": 1, "times": 2},
            "layers": [{"type": "attention", "mixer": m, "mlp": {"kind": "dense", "ff": 64}}] * 2}


@pytest.mark.parametrize("cfg,first", [(latent(16, 512, 64, 100), 500), (latent(24, 260, 10, 0), 300), (latent(16, 256, 32, 333), 650), (latent(128, 60, 4, 64), 80),
                                       (latent(12, 320, 16, 7), 600), (shared(32, 8, 64, 300, 15.0), 300), (shared(18, 6, 128, 0, 0.0), 600),
                                       (shared(40, 2, 48, 129, 3.0), 260)], ids=str)
def test_blocks_match_token_loop(E, cfg, first):
    from lighterpp_b200.models import ARCHITECTURES
    from oracle import kolatar, rutenex
    W = (rutenex if cfg["architecture"] == "Rutenex" else kolatar).random_weights(cfg, 3)
    arch = ARCHITECTURES[cfg["architecture"]]
    c = arch.configure(cfg, 1200)
    engines = [E.Engine(c, "bf16", "f16", flags=f) for f in (0, E.FLAG_NO_PREFILL_GEMM)]
    for e in engines:
        for ours, layer, name, _ in arch.tensors(c):
            e.upload(ours, (np.ascontiguousarray(W[name], dtype=np.float32).view(np.uint32) >> 16).astype(np.uint16), layer)
        e.finalize()
    batched, loop = engines
    toks = np.random.default_rng(4).integers(0, cfg["vocab"], 1024)
    ref = loop.extend(toks, 0, range(1024))

    def check(got, rows):
        want = ref[rows]
        err = np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)
        assert np.isfinite(got).all() and err.max() <= 4e-3, (err.max(), rows[int(err.argmax())])  # the bound of these models' other tests

    for n in (1024, first, first + 1, first + 63, first + 64):  # shorter ones behind stale rows
        check(batched.extend(toks[:n], 0, range(n)), list(range(n)))
    batched.extend(toks[:197], 0)  # a block behind a cache
    check(batched.extend(toks[197:197 + first], 197, range(first)), list(range(197, 197 + first)))
    for e in engines:
        e.close()


def test_sums_over_many_keys_are_not_truncated(E):
    """The tensor cores add with truncation: 3000 alike rows in one accumulator (190 additions of 16 rows, each of which loses half of
    2^-23 of the sum so far on average) come out (190 / 2) 2^-24 = 6e-6 too small.  Rounding errors have no direction, so the error of the
    last 64 tokens' logits is laid onto what a larger attention output would change in them.  64 keys in one accumulator and the value
    and output matrices (64 and 128 inputs) leave 16 additions, 1e-6 at most."""
    from oracle import rutenex
    from rutenex_util import engine
    cfg = latent(8, 64, 16, 0)
    cfg["layers"] = cfg["layers"][:1]
    cfg["layers"][0]["mixer"]["vdim"] = 16
    W = rutenex.random_weights(cfg, 5)
    rng = np.random.default_rng(6)
    W["embed"] = rutenex.bf16_round(rng.standard_normal(136) + 0.2 * rng.standard_normal((320, 136)))
    W["l0.mix.o"] = rutenex.bf16_round(4 * W["l0.mix.o"])
    toks = rng.integers(0, 320, 3072)
    e = engine(E, cfg, W, "bfloat16", 3072)
    got = e.extend(toks, 0, range(3008, 3072)).astype(np.float64)
    e.close()
    want = rutenex.forward(cfg, W, toks)[-64:]
    more = (rutenex.forward(cfg, {**W, "l0.mix.o": W["l0.mix.o"].astype(np.float64) * 1.001}, toks)[-64:] - want) / 1e-3
    short = float(((got - want) * more).sum() / (more * more).sum())
    print("attention output off by", short)
    assert np.linalg.norm(got - want) <= 2e-3 * np.linalg.norm(want) and abs(short) <= 1.5e-6, short
