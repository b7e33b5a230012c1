"""The tensor-core attention of a decode step at the edges of its 16-position steps, of a round of the block's warps and of the ring that the
rows are copied through: splits that the ring holds whole and splits that go through it several times, the current position in each of them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

POSITIONS = (0, 1, 14, 15, 16, 17, 127, 128, 129, 255, 256, 257, 383, 384, 385, 500, 511, 512, 513, 640, 1023, 1024, 1089)


@pytest.mark.parametrize("heads,kv_heads,hs", [(8, 2, 64), (8, 1, 64), (4, 4, 64), (4, 1, 128), (2, 2, 128), (8, 1, 128)])
def test_step_at_edges(oracle, heads, kv_heads, hs):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from lighterpp_b200 import engine as E, synth
    from test_gpu_parity import check_logits
    c, dt, tied, seed = synth.SHAPES["mini-8b-f16"]
    c = type(c)(**{**c.asdict(), "seq_len": 1100, "dim": heads * hs, "n_heads": heads, "n_kv_heads": kv_heads, "n_layers": 1})
    assert c.head_size == hs
    T = synth.gen_model(c, seed, dt, tied)
    rng = np.random.default_rng([heads, kv_heads, hs])
    m = oracle.model(c, synth.as_f32(T))
    ko, vo = m.kv_cache()
    engines = [E.Engine(c, dt, "f16", attn_splits=s) for s in (0, 1, 2)]  # at least four splits of one ring; one split; two
    k, v = (rng.standard_normal((kv_heads, c.seq_len - 1, hs)).astype(np.float16) for _ in range(2))
    ko[0, :, :c.seq_len - 1], vo[0, :, :c.seq_len - 1] = k, v
    for e in engines:
        e.load_weights(T)
        e.kv_prefill(0, k, v, c.seq_len - 1)
    for i, (pos, t) in enumerate(zip(POSITIONS, synth.prompt_tokens(c.vocab_size, len(POSITIONS), seed))):
        ref = m.step_logits(int(t), pos)
        for e in engines:
            check_logits(ref, e.step_logits(int(t), pos), dt)
    for e in engines:
        e.close()
