"""Prompt attention, both kernels (HX_PF_ATTN forces one): the tensor-core kernel with every way a group of heads fills its 128-row tiles,
token counts around row and key tiles, and chunks that begin inside a key tile (HX_PF_CHUNK, in whole groups of 26: 52 and 104); prompts of several chunks.  The K and V
rows of the second layer depend on every token's attention in the first; the logits are checked against the CPU restatement."""
import numpy as np
import pytest

import helix_b200 as hb
import oracle_lib as ol

pytestmark = pytest.mark.gpu


def _model(tmp_path, NH, NKV, DM=256):
    cfg = dict(NL=2, DM=DM, NH=NH, NKV=NKV, DH=128, DFF=256, NV=300)
    path = str(tmp_path / "m.weights")
    ol.write_v3(path, cfg, ol.synth_tensors(cfg, seed=10 * NH + NKV))
    return path


def _prompt(path, ids, monkeypatch, attn, chunk=None):
    monkeypatch.setenv("HX_PF_ATTN", attn)
    if chunk:
        monkeypatch.setenv("HX_PF_CHUNK", str(chunk))
    m = hb.Model.load(path, kv_cap=len(ids) + 4)
    monkeypatch.delenv("HX_PF_ATTN")
    monkeypatch.delenv("HX_PF_CHUNK", raising=False)
    nx, lg = m.prefill(ids, want_logits=True)
    rows = [m.kv_read(1, h, 0, len(ids)) for h in range(m.cfg.n_kv_heads)]
    m.close()
    return nx, lg, rows


def _near(a, b):
    # f32 sums of the same values in another order through one layer
    for x, y in zip(a, b):
        for u, v in zip(x, y):
            assert np.max(np.abs(u - v)) < 1e-4 * max(1.0, float(np.max(np.abs(v))))


@pytest.mark.parametrize("NH,NKV", [(2, 2), (6, 2), (4, 1), (5, 1), (8, 1)])
@pytest.mark.parametrize("T,chunk", [(1, None), (42, None), (43, None), (128, None), (129, None), (257, None), (200, 72), (300, 120)])
def test_tensor_core_kernel(tmp_path, monkeypatch, NH, NKV, T, chunk):
    path = _model(tmp_path, NH, NKV)
    om = ol.OracleModel(path, kv_cap=T + 4)
    ids = np.random.default_rng(T).integers(0, 300, T).astype(np.int32)
    lo = om.prefill(ids)
    nx, lg, rows = _prompt(path, ids, monkeypatch, "tc", chunk)
    assert np.max(np.abs(lo - lg)) < 2e-4 and nx == int(np.argmax(lo))
    _near(rows, _prompt(path, ids, monkeypatch, "vec")[2])
    om.close()


def test_vector_kernel_in_chunks(tmp_path, monkeypatch):
    path = _model(tmp_path, 4, 1)
    ids = np.random.default_rng(5).integers(0, 300, 200).astype(np.int32)
    one, many = _prompt(path, ids, monkeypatch, "vec"), _prompt(path, ids, monkeypatch, "vec", 48)
    assert one[0] == many[0] and np.max(np.abs(one[1] - many[1])) < 2e-4
    _near(one[2], many[2])


def test_prompt_longer_than_a_chunk(tmp_path, monkeypatch):
    """1100 tokens: two chunks of 572 and 528 by the rule that also picks the kernel."""
    path = _model(tmp_path, 4, 1, DM=128)
    om = ol.OracleModel(path, kv_cap=1104)
    ids = np.random.default_rng(6).integers(0, 300, 1100).astype(np.int32)
    lo = om.prefill(ids)
    nx, lg, rows = _prompt(path, ids, monkeypatch, "rule")
    assert np.max(np.abs(lo - lg)) < 2e-4 and nx == int(np.argmax(lo))
    _near(rows, _prompt(path, ids, monkeypatch, "vec", 48)[2])
    om.close()
