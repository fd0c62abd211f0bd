"""The chunk GEMM's kinds (pairs of CTAs, clusters over K, K in several blocks, an odd number of row tiles) at token
counts around its groups of up to 26, through a prompt's logits and cached rows against the CPU restatement.  (The prompt attention
has tests/test_prompt_attention_gpu.py.)"""
import numpy as np
import pytest

import helix_b200 as hb
import oracle_lib as ol

pytestmark = pytest.mark.gpu

# K of 9 and 17 cells of 256 columns, 30 and 68 row tiles, a vocabulary of three tiles
CFG = dict(NL=1, DM=2304, NH=18, NKV=6, DH=128, DFF=4352, NV=300)


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    path = str(tmp_path_factory.mktemp("chunk") / "m.weights")
    ol.write_v3(path, CFG, ol.synth_tensors(CFG, seed=41))
    return path


@pytest.mark.parametrize("T", [1, 24, 25, 26, 27, 52, 53, 130])
def test_prompt_logits_and_cache_rows(model, T):
    om, gm = ol.OracleModel(model, kv_cap=T + 8), hb.Model.load(model, kv_cap=T + 8)
    ids = np.random.default_rng(T).integers(0, CFG["NV"], T).astype(np.int32)
    lo = om.prefill(ids)
    nx, lg = gm.prefill(ids, want_logits=True)
    assert np.max(np.abs(lo - lg)) < 2e-4 and nx == int(np.argmax(lo))
    one = hb.Model.load(model, kv_cap=T + 8)                       # the same rows written token by token
    for p in range(T):
        one.decode_step(int(ids[p]), p)
    for layer, head in ((0, 1), (0, 5)):
        for a, b in zip(gm.kv_read(layer, head, 0, T), one.kv_read(layer, head, 0, T)):
            assert np.max(np.abs(a - b)) < 1e-4 * max(1.0, float(np.max(np.abs(b))))
    om.close(); gm.close(); one.close()


def test_repeated_prompts_are_bit_equal(model):
    """Many units per CTA through the staging and the receive buffer of the cluster's CTAs: what a buffer held for one unit is read before the
    next unit's sums arrive, so a prompt gives the same bits every time."""
    gm = hb.Model.load(model, kv_cap=320)
    ids = np.random.default_rng(7).integers(0, CFG["NV"], 301).astype(np.int32)
    _, want = gm.prefill(ids, want_logits=True)
    rows = gm.kv_read(0, 5, 0, 301)
    for _ in range(40):
        _, lg = gm.prefill(ids, want_logits=True)
        assert np.array_equal(lg.view(np.uint32), want.view(np.uint32))
    for a, b in zip(gm.kv_read(0, 5, 0, 301), rows):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    gm.close()
