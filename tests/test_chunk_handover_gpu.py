"""Hand-overs between the roles of the chunk GEMM where little time lies between them: one to three cells of K per CTA, token groups of two
and of 26, and plans in which a cluster goes from the last tile of a token group to several tiles of the next with fewer cells of K.
A prompt gives the same bits every time, and the K and V rows of the second layer, which depend on every token's sums in the first, are those
of the token-by-token path (f32 sums of the same values in another order through one layer)."""
import numpy as np
import pytest

import helix_b200 as hb

pytestmark = pytest.mark.gpu

SHAPES = {
    "K768": dict(n_layers=2, d_model=768, n_heads=6, n_kv_heads=6, head_dim=128, d_ff=3072, vocab=300),
    "K12288": dict(n_layers=2, d_model=4096, n_heads=32, n_kv_heads=8, head_dim=128, d_ff=12288, vocab=300),
    "K25600": dict(n_layers=2, d_model=5120, n_heads=64, n_kv_heads=8, head_dim=128, d_ff=25600, vocab=300),
}


def _rows(m, T):
    return [a for h in range(m.cfg.n_kv_heads) for a in m.kv_read(1, h, 0, T)]


@pytest.mark.parametrize("shape,T,repeats", [("K768", 2, 60), ("K768", 26, 60), ("K768", 53, 60), ("K768", 300, 40),
                                             ("K12288", 212, 12), ("K12288", 262, 12), ("K25600", 128, 12), ("K25600", 270, 8)])
def test_repeated_prompts_are_bit_equal_and_near_the_token_path(shape, T, repeats):
    ids = np.random.default_rng(T).integers(0, 300, T).astype(np.int32)
    m, one = (hb.Model.synth(SHAPES[shape], seed=T, kv_cap=T + 4) for _ in range(2))
    _, want = m.prefill(ids, want_logits=True)
    rows = _rows(m, T)
    for _ in range(repeats):
        _, lg = m.prefill(ids, want_logits=True)
        assert np.array_equal(lg.view(np.uint32), want.view(np.uint32))
        assert all(np.array_equal(a.view(np.uint32), b.view(np.uint32)) for a, b in zip(_rows(m, T), rows))
    for p in range(T):
        one.decode_step(int(ids[p]), p)
    for a, b in zip(rows, _rows(one, T)):
        assert np.max(np.abs(a - b)) < 1e-4 * max(1.0, float(np.max(np.abs(b))))
    m.close(); one.close()
