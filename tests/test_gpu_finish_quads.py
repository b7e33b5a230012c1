"""Finishing kernels that take four rows of four tokens a thread: prompts whose token counts leave every remainder of four and lie on either
side of where the kernels change, against the token loop; sizes that the quads take (heads, rotated parts and sections on multiples of
four) and sizes that keep the pairs (a rotated part of 6, an odd head, a row total off the multiples of four)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SIZES = (127, 128, 129, 130, 191, 192, 193, 223, 224, 225, 239, 240, 241, 242, 259)


def latent(heads, dim, rot_dim):
    rot = {"base": 1e4, "dims": rot_dim, "scaling": {"factor": 4.0, "original": 64, "fast": 8.0, "slow": 1.0}}
    mix = {"heads": heads, "dim": dim, "rot_dim": rot_dim, "vdim": 24, "kv_rank": 72, "scale": 56 ** -0.5, "mask": {"size": 100}, "rot": rot}
    return {"architecture": "Rutenex", "width": 136, "vocab": 320, "norm": {"eps": 1e-5},
            "layers": [{"type": "latent_attention", "mixer": mix, "mlp": {"kind": "dense", "ff": 200}}] * 2}


def shared(dim, dims):
    rot = {"base": 1e4, "dims": dims, "scaling": {"factor": 4.0, "original": 64, "fast": 8.0, "slow": 1.0}}
    attn = {"type": "attention", "mlp": {"kind": "dense", "ff": 200},
            "mixer": {"heads": 4, "kv_heads": 2, "dim": dim, "vdim": dim, "scale": dim ** -0.5, "softcap": 15.0, "mask": {"size": 130}, "rot": rot}}
    return {"architecture": "Kolatar", "width": 112, "vocab": 300, "norm": {"eps": 1e-5}, "embedding": {"scale": 10.0}, "logit_scale": 1.5,
            "loop": {"start": 0, "stop": 1, "times": 2}, "layers": [attn, attn]}


def takes_quads(cfg):
    """What the host asks of a model's sizes before it launches the kernels that take four rows a thread."""
    mix = cfg["layers"][0]["mixer"]
    if cfg["architecture"] == "Kolatar":
        return mix["dim"] % 4 == 0 and mix["rot"]["dims"] % 4 == 0
    even = lambda n: n + n % 2
    rows = even(mix["heads"] * mix["dim"]) + mix["heads"] * mix["rot_dim"] + even(mix["kv_rank"]) + mix["rot_dim"] + even(mix["heads"])
    return mix["dim"] % 4 == 0 and mix["rot_dim"] % 4 == 0 and rows % 4 == 0


@pytest.mark.parametrize("cfg,quads", [(latent(8, 40, 16), True), (latent(6, 40, 16), False), (latent(8, 40, 6), False), (shared(48, 16), True),
                                       (shared(48, 6), False), (shared(33, 16), False)],
                         ids=["latent", "latent-rows-off-four", "latent-pairs", "shared", "shared-pairs", "shared-odd"])
def test_blocks_match_the_token_loop(cfg, quads):
    assert takes_quads(cfg) == quads  # every case stays on the kernel that it is named for
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from lighterpp_b200 import engine as E
    from lighterpp_b200.models import ARCHITECTURES
    from oracle import kolatar, rutenex
    W = (rutenex if cfg["architecture"] == "Rutenex" else kolatar).random_weights(cfg, 3)
    arch = ARCHITECTURES[cfg["architecture"]]
    c = arch.configure(cfg, 300)
    engines = [E.Engine(c, "bf16", "f16", flags=f) for f in (0, E.FLAG_NO_PREFILL_GEMM)]
    for e in engines:
        for ours, layer, name, _ in arch.tensors(c):
            e.upload(ours, (np.ascontiguousarray(W[name], dtype=np.float32).view(np.uint32) >> 16).astype(np.uint16), layer)
        e.finalize()
    toks = np.random.default_rng(4).integers(0, cfg["vocab"], 300)
    ref = engines[1].extend(toks, 0, range(300))
    for n in SIZES:
        got = engines[0].extend(toks[:n], 0, range(n))
        err = np.linalg.norm(got - ref[:n], axis=1) / np.linalg.norm(ref[:n], axis=1)
        assert np.isfinite(got).all() and err.max() <= 4e-3, (n, err.max())  # the bound of these models' other tests
    for e in engines:
        e.close()
