"""Infinities and NaN in the activations of the chunk path: digits cannot spell them, the outputs of the token show them (as the CPU
restatement's do), and other tokens of the same launch are not touched."""
import numpy as np
import pytest

import helix_b200 as hb
import oracle_lib as ol

pytestmark = pytest.mark.gpu
CFG = dict(NL=2, DM=256, NH=4, NKV=2, DH=64, DFF=512, NV=300)
BAD = 7


def _model(tmp_path, change, **kw):
    t = ol.synth_tensors(CFG, seed=17)
    change(t)
    path = str(tmp_path / "m.weights")
    ol.write_v3(path, CFG, t)
    return ol.OracleModel(path, kv_cap=64), hb.Model.load(path, kv_cap=64, **kw)


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_embedding_row_behind_a_norm(tmp_path, value):
    def change(t):
        t["model.embed_tokens.weight"][BAD, 100] = value
    om, gm = _model(tmp_path, change, batch=3)
    ids = np.array([3, 4, 5, 6, 8], np.int32)
    lo = om.prefill(ids)
    nx, lg = gm.prefill(ids, want_logits=True)
    assert np.max(np.abs(lo - lg)) < 2e-4 and nx == int(np.argmax(lo))
    bad = np.array([3, 4, BAD, 6, 8], np.int32)
    lg = gm.prefill(bad, want_logits=True)[1]
    assert np.isnan(om.prefill(bad)).all() and np.isnan(lg).all()
    # a batch step: the sequences beside it keep their tokens
    pos = np.zeros(3, np.int32)
    want = gm.decode_batch(np.array([3, 9, 11], np.int32), pos)
    got = gm.decode_batch(np.array([3, BAD, 11], np.int32), pos)
    assert got[0] == want[0] and got[2] == want[2]
    om.close(); gm.close()


@pytest.mark.parametrize("T", [2, 30])
def test_hidden_vector_that_overflows(tmp_path, T):
    """gate and up of 1e20 times the usual size: their product is infinite, and no norm stands before the down projection."""
    def change(t):
        for k in t:
            if "gate_proj" in k or "up_proj" in k:
                t[k] *= np.float32(1e20)
    om, gm = _model(tmp_path, change)
    ids = np.random.default_rng(T).integers(0, 300, T).astype(np.int32)
    lg = gm.prefill(ids, want_logits=True)[1]
    assert not np.isfinite(om.prefill(ids)).any() and np.isnan(lg).all()
    om.close(); gm.close()
