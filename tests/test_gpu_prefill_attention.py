"""Causal attention of prompt blocks (128 rows = tokens x query heads of a group, 128 keys a tile) against the token loop: both
head sizes, groups that do and do not divide a row tile, token counts around row and key tiles, blocks whose keys one CTA or a
cluster takes, and whatever a cache holds behind the block."""
import numpy as np
import pytest

from lighterpp_b200 import synth
from lighterpp_b200.formats import ModelConfig

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def E():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from lighterpp_b200 import engine
    return engine


# head size 64 with groups of 8, 3 and 1, head size 128 with groups of 4, 7 and 1
@pytest.mark.parametrize("dim,heads,kv", [(512, 8, 1), (384, 6, 2), (256, 4, 4), (1024, 8, 2), (896, 7, 1), (256, 2, 2)])
def test_blocks_match_token_loop(E, dim, heads, kv):
    c = ModelConfig(dim, 256, 2, heads, kv, 320, 1536, 10000.0)
    T = synth.gen_model(c, 7, "f16", True)
    # q . k / sqrt(head size) has a spread of (2 x 0.02)^2 dim = 0.4 to 1.6.  Rounding the queries to FP16 (2^-11) moves scores and with
    # them the probabilities by 2^-11 of that, under 8e-4; rounded probabilities and cache rows add 2^-11 each.  (At four times 0.02
    # the spread is 6.6 for the width of 1024 and the first of these alone over 3e-3: seen there.)
    for l in range(c.n_layers):
        T["wq"][l] = (T["wq"][l].astype(np.float32) * 2).astype(np.float16)
        T["wk"][l] = (T["wk"][l].astype(np.float32) * 2).astype(np.float16)
    toks = synth.prompt_tokens(c.vocab_size, 1500, 7)
    batched, loop = E.Engine(c, "f16", "f16"), E.Engine(c, "f16", "f16", flags=E.FLAG_NO_PREFILL_GEMM)
    for e in (batched, loop):
        e.load_weights(T)
    stale = np.full((kv, c.seq_len, c.head_size), np.inf, np.float16)
    stale[:, ::2] = np.nan
    sizes = (2, 15, 16, 17, 33, 64, 127, 128, 129, 255, 257, 640, 1300)
    ends = sorted({n - 1 for n in sizes} | {1499})
    ref = loop.extend(toks, 0, ends)

    def check(got, row):
        want = ref[ends.index(row)]
        assert np.isfinite(got).all() and np.linalg.norm(got - want) <= 2e-3 * np.linalg.norm(want), (row, np.linalg.norm(got - want) / np.linalg.norm(want))

    for n in sizes:
        for l in range(c.n_layers):
            batched.kv_prefill(l, stale, stale, c.seq_len)
        check(batched.extend(toks[:n], 0, [n - 1])[0], n - 1)
    for first, n in ((127, 2), (640, 17), (1000, 300), (1300, 200), (1483, 17)):  # behind a cache
        for l in range(c.n_layers):
            batched.kv_prefill(l, stale, stale, c.seq_len)
        batched.extend(toks[:first], 0)
        end = first + n - 1
        got = batched.extend(toks[first:first + n], first, [n - 1])[0]
        if end in ends:
            check(got, end)
        else:
            check(batched.extend(toks[end + 1:1500], end + 1, [1498 - end])[0], 1499)
    for e in (batched, loop):
        e.close()
