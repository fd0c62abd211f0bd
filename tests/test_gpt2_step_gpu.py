"""GPT-2 prompts through the chunk GEMM and tokens through the one-launch layer kernel (d_model 256, 512 and 768), against the
fp32 CPU restatement: contexts around the kernel's passes of 256 keys and beyond two of them, the first position, and the last of the cache."""
import numpy as np
import pytest

import helix_b200 as hb
from test_gpt2_gpu import OracleGpt2, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d_model,n_layers,T,cap", [(256, 3, 1, 40), (256, 2, 126, 136), (512, 2, 25, 40), (768, 2, 255, 262), (256, 2, 510, 520), (512, 2, 34, 40)])
def test_prompt_then_tokens_match_checker(d_model, n_layers, T, cap):
    shape = dict(n_layers=n_layers, d_model=d_model, n_heads=d_model // 64, d_ff=4 * d_model, vocab=517, max_ctx=cap)
    wt = synth(shape, d_model + T)
    om = OracleGpt2(shape, wt, cap)
    gm = hb.Model.gpt2(shape, wt, kv_cap=cap)
    ids = np.random.default_rng(T).integers(0, shape["vocab"], T).astype(np.int32)
    for p in range(T):
        want = om.decode(ids[p], p)
    tok, lg = gm.prefill(ids, want_logits=True)
    assert np.max(np.abs(lg - want)) < 2e-4 and tok == int(np.argmax(want))
    for p in range(T, min(cap, T + 6)):
        want = om.decode(tok, p)
        tok, lg = gm.decode_step(tok, p, want_logits=True)
        assert np.max(np.abs(lg - want)) < 2e-4, p
        assert tok == int(np.argmax(want))
    gm.close()


@pytest.mark.parametrize("d_model", [256, 768])
def test_profiled_steps_run_op_by_op_with_the_same_tokens(d_model):
    """The layers' dense layout is made from the layer kernel's cells when profiling asks for it."""
    shape = dict(n_layers=2, d_model=d_model, n_heads=d_model // 64, d_ff=4 * d_model, vocab=517, max_ctx=40)
    wt = synth(shape, d_model)
    om, gm = OracleGpt2(shape, wt, 40), hb.Model.gpt2(shape, wt, kv_cap=40)
    tok, want = 11, []
    for p in range(8):
        tok = int(np.argmax(om.decode(tok, p))); want.append(tok)
    assert list(gm.decode_loop(11, 0, 8)[0]) == want
    gm.set_profile(True)
    assert list(gm.decode_loop(11, 0, 8)[0]) == want
    st = gm.last_stats()
    assert st["ms_gemv"] > 0 and st["ms_attn"] > 0
    gm.set_profile(False)
    assert list(gm.decode_loop(11, 0, 8)[0]) == want
    gm.close()
