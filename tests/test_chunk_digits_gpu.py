"""The digits of the chunk path (eight base-13 digits per activation, a scale per block of 32 columns of K) at the edges of its token groups and
of a block's scale range: a prompt's logits against the CPU restatement, and one linear by itself -- the V rows of the first layer are
W_v RMSNorm(embedding), nothing else -- against 64 bits."""
import numpy as np
import pytest

import helix_b200 as hb
import oracle_lib as ol

pytestmark = pytest.mark.gpu
TOL = 2e-4
# K of 3 and 17 cells of 256 columns, the last one ragged
CFG = dict(NL=2, DM=640, NH=5, NKV=5, DH=128, DFF=4200, NV=300)


def _check(om, gm, one, ids):
    """Logits against the CPU restatement; the second layer's K and V rows, which depend on all outputs of every token in the first, against the
    token-by-token path (f32 sums of the same values in another order through one layer)."""
    T = len(ids)
    lo = om.prefill(ids)
    nx, lg = gm.prefill(ids, want_logits=True)
    assert np.max(np.abs(lo - lg)) < TOL and nx == int(np.argmax(lo))
    for p in range(T):
        one.decode_step(int(ids[p]), p)
    for h in range(CFG["NKV"]):
        for a, b in zip(gm.kv_read(1, h, 0, T), one.kv_read(1, h, 0, T)):
            assert np.max(np.abs(a - b)) < 1e-4 * max(1.0, float(np.max(np.abs(b))))


@pytest.fixture(scope="module")
def plain(tmp_path_factory):
    path = str(tmp_path_factory.mktemp("digits") / "m.weights")
    ol.write_v3(path, CFG, ol.synth_tensors(CFG, seed=7))
    om, gm, one = ol.OracleModel(path, kv_cap=464), hb.Model.load(path, kv_cap=464), hb.Model.load(path, kv_cap=464)
    yield om, gm, one
    om.close(); gm.close(); one.close()


# groups of at most 26 tokens, all of one even size: one token, a pair and its half, full groups, one token more, odd remainders; 449: the
# digit kernel of long chunks for the hidden vector (two slices of 4096 columns a token)
@pytest.mark.parametrize("T", [1, 2, 3, 25, 26, 27, 52, 53, 79, 105, 225, 449])
def test_group_edges(plain, T):
    _check(*plain, np.random.default_rng(T).integers(0, CFG["NV"], T).astype(np.int32))


# one element `ratio` times the others: the blocks without it have their own scale down to 2^-9 of the vector's and no further
@pytest.mark.parametrize("ratio", [2.0, 64.0, 512.0, 1024.0, 1e6])
def test_blocks_far_below_the_largest_element(tmp_path, ratio):
    t = ol.synth_tensors(CFG, seed=9)
    e = t["model.embed_tokens.weight"]
    e[::2, 300] = np.float32(np.abs(e).max() * ratio)      # second of three cells
    e[1::2, 5] = np.float32(-np.abs(e[1::2]).max() * ratio)
    e[:, 512:] = 0                                          # a cell of zeros
    path = str(tmp_path / "m.weights")
    ol.write_v3(path, CFG, t)
    om, gm, one = ol.OracleModel(path, kv_cap=64), hb.Model.load(path, kv_cap=64), hb.Model.load(path, kv_cap=64)
    _check(om, gm, one, np.random.default_rng(3).integers(0, CFG["NV"], 41).astype(np.int32))
    om.close(); gm.close(); one.close()


def _block_units(x):
    """What the digits of a vector resolve, element by element: 2^-27 of the power of two at or below the block's largest one, and at least 2^-36 of
    the vector's.  A block: 16 columns of a 64-column step of K and the 16 at the same place of the other step of the same 128."""
    K = (len(x) + 255) // 256 * 256
    a = np.zeros(K)
    a[:len(x)] = np.abs(x)
    a = a.reshape(K // 128, 2, 4, 16)
    p2 = lambda m: 2.0 ** np.floor(np.log2(np.maximum(m * 1.000001, 1e-30)))       # (a power of two may be passed in f32)
    s = np.maximum(p2(a.max(axis=(1, 3), keepdims=True)), p2(a.max()) * 2.0 ** -9)
    return (np.broadcast_to(s, a.shape) * 2.0 ** -27).reshape(K)[:len(x)]


# T: groups up to 16 tokens (their column scales lie closer) and wider ones, several groups, both sides of the line to the
# kernel of long chunks
@pytest.mark.parametrize("DM,T", [(768, 6), (1024, 16), (1024, 18), (1024, 53), (4096, 7), (4096, 26), (4096, 450), (8192, 444), (8192, 446)])
def test_a_linear_against_64_bits(tmp_path, DM, T):
    """2-norm over the rows of a token.  Rows with weight on the vector's large element: below one unit of an f32, 2^-23, for every vector (an element times
    the norm's factor, the fold of the digits and the sums round; 5e-8 to 1e-7 seen).  Rows without: what the digits of the other elements resolve comes on
    top (every element off by up to half of its unit: 1/sqrt(12) of it in the mean; 1.5 for few elements)."""
    rng = np.random.default_rng(DM + T)
    cfg = dict(NL=1, DM=DM, NH=2, NKV=2, DH=128, DFF=256, NV=T)
    big = DM // 3
    x = rng.standard_normal((T, DM))
    for t in range(T):
        if t % 6 == 1:
            x[t] = rng.standard_t(3, DM)
        if t % 6 >= 2:
            x[t, big] = 4.0 * (2.0, 64.0, 1000.0, 1e6)[t % 6 - 2]
    x = x.astype(np.float32)
    w = 0.02 * rng.standard_normal((256, DM))
    w[128:, big] = 0.0
    t = ol.synth_tensors(cfg, seed=1)
    t["model.embed_tokens.weight"], t["model.layers.0.self_attn.v_proj.weight"] = x, w.astype(np.float32)
    t["model.layers.0.input_layernorm.weight"] = np.ones(DM, np.float32)
    path = str(tmp_path / "m.weights")
    ol.write_v3(path, cfg, t)
    m = hb.Model.load(path, kv_cap=T + 4)
    m.prefill(np.arange(T, dtype=np.int32))
    got = np.concatenate([m.kv_read(0, h, 0, T)[1].reshape(T, 128) for h in range(2)], axis=1).astype(np.float64)
    m.close()
    words, micro, ts, _ = ol.quantize(w.astype(np.float32))
    w64 = ol.dequant_micro(words, micro, 1.0)[:, :DM].astype(np.float64) * ts
    assert not w64[128:, big].any()
    for t in range(T):
        v = x[t].astype(np.float64)
        v /= np.sqrt(np.mean(v * v) + 1e-5)
        digits = np.sum(_block_units(v) ** 2) / 12
        for rows, extra in ((slice(0, 128), 0.0), (slice(128, 256), digits / (v @ v - v[big] ** 2))):
            want, have = w64[rows] @ v, got[t, rows]
            have = have * (want @ want) / (want @ have)      # the norm's factor, one f32 number per token, is not the linear's
            assert np.linalg.norm(have - want) < np.sqrt(2.0 ** -46 + 2.25 * extra) * np.linalg.norm(want), (t, rows)
