"""The chunk path's buffers when device memory is short: a prompt makes do with smaller chunks, a failed attempt is reported and
leaves a model that works once there is room again."""
import numpy as np
import pytest
import torch

import helix_b200 as hb
import oracle_lib as ol

pytestmark = pytest.mark.gpu
HX_ERR_NOMEM = 6
# wide hidden layer: 43 MB of chunk buffers at 78 tokens, 71 at 130, 142 at 260, 567 at 1040
CFG = dict(NL=1, DM=512, NH=4, NKV=4, DH=128, DFF=32768, NV=300)


def _leave(mib):
    free = torch.cuda.mem_get_info()[0]
    return torch.empty(free - (mib << 20), dtype=torch.uint8, device="cuda")


@pytest.fixture(scope="module")
def path(tmp_path_factory, tiny_file):
    torch.zeros(1, device="cuda")
    m = hb.Model.load(tiny_file, kv_cap=64, batch=2)      # the kernels are loaded before memory gets short
    m.prefill(np.arange(40, dtype=np.int32)); m.decode_batch(np.zeros(2, np.int32), np.zeros(2, np.int32)); m.close()
    p = str(tmp_path_factory.mktemp("wide") / "m.weights")
    ol.write_v3(p, CFG, ol.synth_tensors(CFG, seed=5))
    return p


@pytest.mark.parametrize("mib,fits", [(130, True), (32, False)])
def test_prompt_with_little_memory(path, mib, fits):
    om, gm = ol.OracleModel(path, kv_cap=1100), hb.Model.load(path, kv_cap=1100, batch=2)
    ids = np.random.default_rng(1).integers(0, 300, 150).astype(np.int32)
    want = om.prefill(ids)
    hog = _leave(mib)
    try:
        if not fits:
            for call in (lambda: gm.prefill(ids), lambda: gm.prefill(ids), lambda: gm.decode_batch(ids[:2], np.zeros(2, np.int32))):
                with pytest.raises(hb.HxError) as e:
                    call()
                assert e.value.code == HX_ERR_NOMEM
            del hog
            torch.cuda.empty_cache()
        for _ in range(2):
            nx, lg = gm.prefill(ids, want_logits=True)
            assert np.max(np.abs(lg - want)) < 2e-4 and nx == int(np.argmax(want))
    finally:
        hog = None
        torch.cuda.empty_cache()
        om.close(); gm.close()


def test_batch_step_then_longer_prompts_then_the_captured_step(gqa4_file):
    """The buffers of a batch step grow for a prompt; the step captured on the old ones is captured again."""
    gm, one = hb.Model.load(gqa4_file, kv_cap=200, batch=3), hb.Model.load(gqa4_file, kv_cap=200)
    rng = np.random.default_rng(2)
    prompts = [rng.integers(0, 300, 150).astype(np.int32) for _ in range(3)]
    gm.decode_batch_loop(np.array([1, 2, 3], np.int32), 0, 3)
    first = np.array([gm.prefill_seq(s, p) for s, p in enumerate(prompts)], np.int32)
    got = gm.decode_batch_loop(first, 150, 4)[0]
    for s, p in enumerate(prompts):
        assert list(one.generate(p, 5)[0]) == [first[s]] + list(got[:, s])
    gm.close(); one.close()


def test_a_failed_allocation_is_not_reported_again_by_the_next_call(tiny_file):
    with pytest.raises(hb.HxError) as e:
        hb.Model.load(tiny_file, kv_cap=1 << 30)              # a KV cache larger than the device
    assert e.value.code == HX_ERR_NOMEM
    w = np.random.default_rng(0).standard_normal((48, 1000)).astype(np.float32)
    assert np.array_equal(hb.quantize_host(w)[0], ol.quantize(w)[0])
