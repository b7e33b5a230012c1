"""Decoding with a cluster of CTAs per head against the double-precision statement: one to many heads (clusters of eight and of four, more
heads than either takes), fewer keys than CTAs, windows that slide and none, latents and parts off every multiple, and portions before
and after single steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,dim,rot,vdim,rank,window", [(1, 16, 16, 8, 16, 5), (3, 40, 6, 23, 72, 30), (16, 64, 32, 64, 256, 64), (18, 24, 8, 16, 100, 17), (19, 24, 8, 16, 100, 17),
                                                           (37, 8, 4, 6, 33, 0), (38, 8, 4, 6, 33, 9), (4, 136, 16, 130, 300, 0)])
def test_steps_match_the_statement(heads, dim, rot, vdim, rank, window):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from lighterpp_b200 import engine as E
    from lighterpp_b200.models import ARCHITECTURES
    from oracle import rutenex
    turns = {"base": 1e4, "dims": rot, "scaling": {"factor": 4.0, "original": 64, "fast": 8.0, "slow": 1.0}}
    mix = {"heads": heads, "dim": dim, "rot_dim": rot, "vdim": vdim, "kv_rank": rank, "scale": (dim + rot) ** -0.5, "rot": turns}
    if window:
        mix["mask"] = {"size": window}
    cfg = {"architecture": "Rutenex", "width": 136, "vocab": 320, "norm": {"eps": 1e-5},
           "layers": [{"type": "latent_attention", "mixer": mix, "mlp": {"kind": "dense", "ff": 200}}] * 2}
    W, arch = rutenex.random_weights(cfg, 3), ARCHITECTURES["Rutenex"]
    c = arch.configure(cfg, 100)
    e = E.Engine(c, "bf16", "f16")
    for ours, layer, name, _ in arch.tensors(c):
        e.upload(ours, (np.ascontiguousarray(W[name], dtype=np.float32).view(np.uint32) >> 16).astype(np.uint16), layer)
    e.finalize()
    toks = np.random.default_rng(4).integers(0, 320, 90)
    ref = rutenex.forward(cfg, W, toks)
    got = np.concatenate([e.extend(toks[p:p + 1], p, [0]) for p in range(40)] + [e.extend(toks[40:70], 40, range(30))] +
                         [e.extend(toks[p:p + 1], p, [0]) for p in range(70, 90)])
    err = np.linalg.norm(got - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert np.isfinite(got).all() and err.max() < 4e-3, (err.max(), int(err.argmax()))  # the bound of this design's other tests
    e.close()
