"""Decode attention around the edges of its ring tiles (36 rows of 128 dimensions per slot, four slots a tile) for every way a
group of heads is folded, and the q/k kernel of a prompt chunk at each head size, against the CPU restatement."""
import numpy as np
import pytest

import helix_b200 as hb
import oracle_lib as ol

pytestmark = pytest.mark.gpu


def _model(tmp_path, NH, NKV, DH):
    cfg = dict(NL=1, DM=256, NH=NH, NKV=NKV, DH=DH, DFF=256, NV=300)
    path = str(tmp_path / "m.weights")
    ol.write_v3(path, cfg, ol.synth_tensors(cfg, seed=NH + DH))
    return path


@pytest.mark.parametrize("NH,NKV,DH", [(2, 2, 128), (5, 1, 128), (8, 1, 128), (6, 2, 64), (7, 1, 32)])
def test_decode_logits_at_tile_edges(tmp_path, monkeypatch, NH, NKV, DH):
    monkeypatch.setenv("HX_ATT_SPLIT", "1")        # one CTA per kv head sees all rows: several tiles
    path, T = _model(tmp_path, NH, NKV, DH), 300
    om, gm = ol.OracleModel(path, kv_cap=T + 4), hb.Model.load(path, kv_cap=T + 4)
    ids = np.random.default_rng(DH).integers(0, 300, T).astype(np.int32)
    for p in range(T):
        want = p in (0, 35, 36, 37, 143, 144, 145, 159, 160, 288, 299)
        got = gm.decode_step(int(ids[p]), p, want_logits=want)
        if want:
            lo = om.prefill(ids[:p + 1])
            assert np.max(np.abs(lo - got[1])) < 2e-4, p
    om.close(); gm.close()


@pytest.mark.parametrize("NH,NKV,DH", [(4, 2, 32), (4, 1, 64), (2, 1, 128), (2, 1, 256)])
def test_prompt_logits_per_head_size(tmp_path, NH, NKV, DH):
    path, T = _model(tmp_path, NH, NKV, DH), 31
    om, gm = ol.OracleModel(path, kv_cap=T + 4), hb.Model.load(path, kv_cap=T + 4)
    ids = np.random.default_rng(DH).integers(0, 300, T).astype(np.int32)
    lo = om.prefill(ids)
    nx, lg = gm.prefill(ids, want_logits=True)
    assert np.max(np.abs(lo - lg)) < 2e-4 and nx == int(np.argmax(lo))
    om.close(); gm.close()
