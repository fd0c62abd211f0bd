"""What this library is used for, as cases that can be timed and compared.

Every case is one call (or one short greedy loop) through the public entry points of helix_b200, at sizes from the
repository's own configurations: the 12288 x 4096 single-matrix round trip, GPT-2 124M with a 32-token prompt and 128 new
tokens, the Qwen3-8B shape at batch 1 and with 64 sequences of 2048 positions, the Qwen3-32B shape at a 4096-position
context.  Weights are seeded synthetic ones (N(0, 0.02), the distribution the benchmark uses), token ids are uniform.

Kinds:
  quantize    device f32 matrix -> words, micro bytes, collapsed scales, tensor scale (the layout the file carries)
  import      the same on host buffers: the call a checkpoint importer makes for every tensor
  dequantize  the packed layout back to f32
  gpt2        GPT-2 124M greedy generation: prompt and new tokens
  step        one token of one sequence with its logits: what a serve loop with a sampler calls
  loop        a greedy loop of a few tokens that stay on the GPU
  prefill     a prompt into the KV cache, logits of its last position
  batch       decode of several sequences that share the weights: all at one position (loop) or each at its own (one call)
"""
import math

import numpy as np
import torch

import helix_b200 as hb
from helix_b200.lib import check

SHAPES = {"8b": hb.QWEN3_8B, "32b": hb.QWEN3_32B}
GPT2 = hb.GPT2_124M
MATRIX = 12288 * 4096          # elements of the largest matrix quantized here
PROMPT = 2048                  # longest prompt


def listed():
    return [
        # a small tensor with a ragged width: the launches are the cost
        {"name": "quantize 48x1000", "kind": "quantize", "rows": 48, "K": 1000},
        # the single-matrix configuration; gate, up and down of the 8B shape
        {"name": "quantize 12288x4096", "kind": "quantize", "rows": 12288, "K": 4096},
        # an o_proj of the 8B shape as the importer hands it over: pageable host memory in and out
        {"name": "import 4096x4096", "kind": "import", "rows": 4096, "K": 4096},
        # a down_proj of the 8B shape, read back
        {"name": "dequantize 4096x12288", "kind": "dequantize", "rows": 4096, "K": 12288},
        # the small-model configuration: latency per token, 160 tokens in a row
        {"name": "gpt2 32+128", "kind": "gpt2", "T": 32, "n_new": 128},
        # the headline configuration halfway through its 256 new tokens
        {"name": "step 8b at 640", "kind": "step", "shape": "8b", "ctx": 640},
        # the largest model on one GPU, long context
        {"name": "loop 32b at 4096", "kind": "loop", "shape": "32b", "ctx": 4096, "n_new": 8},
        # a chat-sized prompt that fills no whole number of chunks
        {"name": "prefill 8b 77", "kind": "prefill", "shape": "8b", "T": 77},
        # the headline configuration's prompt
        {"name": "prefill 8b 512", "kind": "prefill", "shape": "8b", "T": 512},
        # a prompt of the batched configuration
        {"name": "prefill 8b 2048", "kind": "prefill", "shape": "8b", "T": 2048},
        # a lightly loaded server: five requests, each at its own position
        {"name": "batch 8b 5 ragged to 900", "kind": "batch", "shape": "8b", "n_seq": 5, "ctx": 900, "ragged": True, "n_new": 1},
        # the batched configuration: 64 sequences behind 2048-token prompts
        {"name": "batch 8b 64 at 2048", "kind": "batch", "shape": "8b", "n_seq": 64, "ctx": 2048, "ragged": False, "n_new": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["quantize", "import", "dequantize", "gpt2", "step", "loop", "prefill", "prefill", "batch", "batch"])
    if kind in ("quantize", "import", "dequantize"):
        K = _log(rng, 64, 12288)
        n = _log(rng, 1 << 12, MATRIX)
        return {"kind": kind, "rows": max(1, n // K), "K": K}
    if kind == "gpt2":
        return {"kind": kind, "T": _log(rng, 4, 256), "n_new": _log(rng, 8, 128)}
    if kind == "step":
        return {"kind": kind, "shape": rng.choice(["8b", "8b", "32b"]), "ctx": _log(rng, 16, 4096)}
    if kind == "loop":
        return {"kind": kind, "shape": rng.choice(["8b", "8b", "32b"]), "ctx": _log(rng, 16, 4096), "n_new": rng.randint(2, 16)}
    if kind == "prefill":
        return {"kind": kind, "shape": "8b", "T": _log(rng, 8, PROMPT)}
    ragged = rng.random() < 0.5
    return {"kind": kind, "shape": "8b", "n_seq": _log(rng, 2, 64), "ctx": _log(rng, 32, 2048), "ragged": ragged, "n_new": 1 if ragged else rng.randint(2, 4)}


# ---- inputs -------------------------------------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _weights(rows, K, seed):
    """N(0, 0.02) with a few outlier rows, as trained matrices have them: block scales spread over several binades."""
    g = _gen(seed)
    w = torch.randn((rows, K), generator=g, device="cuda") * 0.02
    w[torch.rand((rows,), generator=g, device="cuda") < 0.01] *= 8.0
    return w


def _packed_buffers(rows, K):
    kp = hb.lib().hx_kpad(K)
    return (torch.empty((rows, kp // 7), dtype=torch.int32, device="cuda"), torch.empty((rows, kp // 16), dtype=torch.uint8, device="cuda"),
            torch.empty((rows, kp // 16), dtype=torch.float32, device="cuda"), torch.empty((1,), dtype=torch.float32, device="cuda"))


def _quantize(w, rows, K, words, micro, sc, ts):
    check(hb.lib().hx_quantize_nvfp4(w.data_ptr(), rows, K, words.data_ptr(), micro.data_ptr(), sc.data_ptr(), ts.data_ptr(),
                                     torch.cuda.current_stream().cuda_stream))


def _gpt2_weights(seed):
    g = _gen(seed)
    dm, dff, nv, ctx = GPT2["d_model"], GPT2["d_ff"], GPT2["vocab"], GPT2["max_ctx"]

    def normal(*shape):
        return (torch.randn(shape, generator=g, device="cuda") * 0.02).cpu().numpy()

    def gain():
        return (1.0 + torch.randn((dm,), generator=g, device="cuda") * 0.05).cpu().numpy()

    layers = [dict(ln1_g=gain(), ln1_b=normal(dm), w_qkv=normal(3 * dm, dm), b_qkv=normal(3 * dm), w_proj=normal(dm, dm), b_proj=normal(dm),
                   ln2_g=gain(), ln2_b=normal(dm), w_fc=normal(dff, dm), b_fc=normal(dff), w_proj2=normal(dm, dff), b_proj2=normal(dm))
              for _ in range(GPT2["n_layers"])]
    return dict(wte=normal(nv, dm), wpe=normal(ctx, dm), lnf_g=gain(), lnf_b=normal(dm), layers=layers)


def _capacity(n):
    return (n + 63) // 64 * 64


class State:
    def __init__(self, case):
        self.case = case
        self.kind = case["kind"]


def prepare(case, seed):
    s = State(case)
    kind = s.kind
    rng = np.random.default_rng(seed)
    if kind in ("quantize", "dequantize"):
        s.w = _weights(case["rows"], case["K"], seed)
        s.out = _packed_buffers(case["rows"], case["K"])
        if kind == "dequantize":
            _quantize(s.w, case["rows"], case["K"], *s.out)
            s.kpad = hb.lib().hx_kpad(case["K"])
            s.w = torch.empty((case["rows"], s.kpad), dtype=torch.float32, device="cuda")
    elif kind == "import":
        s.w = _weights(case["rows"], case["K"], seed).cpu().numpy()
    elif kind == "gpt2":
        s.model = hb.Model.gpt2(GPT2, _gpt2_weights(seed), kv_cap=_capacity(case["T"] + case["n_new"]))
        s.prompt = rng.integers(0, GPT2["vocab"], case["T"]).astype(np.int32)
    else:
        shape = SHAPES[case["shape"]]
        nv = shape["vocab"]
        if kind == "prefill":
            s.model = hb.Model.synth(shape, seed=seed, kv_cap=_capacity(case["T"]))
            s.prompt = rng.integers(0, nv, case["T"]).astype(np.int32)
        elif kind in ("step", "loop"):
            s.model = hb.Model.synth(shape, seed=seed, kv_cap=_capacity(case["ctx"] + case.get("n_new", 1)))
            s.model.fill_kv(case["ctx"], seed)
            s.tok = int(rng.integers(0, nv))
            if kind == "step":      # page-locked, as a loop that calls once per token keeps them
                s.logits, s.io = hb.PinnedArray(nv), hb.PinnedArray(2, np.int32)
        else:
            n = case["n_seq"]
            s.model = hb.Model.synth(shape, seed=seed, kv_cap=_capacity(case["ctx"] + case["n_new"]), batch=n)
            s.model.fill_kv(case["ctx"], seed)
            s.ids = rng.integers(0, nv, n).astype(np.int32)
            s.pos = rng.integers(0, case["ctx"] + 1, n).astype(np.int32)
    return s


# ---- one pass -----------------------------------------------------------------------------------------------------


def _last_head(model, seq, pos, n):
    """K and V rows that a pass left in the last layer's last head: a part of the state that depends on every layer."""
    return model.kv_read(model.cfg.n_layers - 1, model.cfg.n_kv_heads - 1, pos, n, seq=seq)


def run(s):
    c = s.case
    if s.kind == "quantize":
        _quantize(s.w, c["rows"], c["K"], *s.out)
        return s.out
    if s.kind == "import":
        return hb.quantize_host(s.w)
    if s.kind == "dequantize":
        words, micro, _, ts = s.out
        check(hb.lib().hx_dequant_nvfp4(words.data_ptr(), micro.data_ptr(), ts.data_ptr(), None, s.w.data_ptr(), c["rows"], s.kpad,
                                        torch.cuda.current_stream().cuda_stream))
        return s.w
    if s.kind == "gpt2":
        ids = s.model.generate(s.prompt, c["n_new"])[0]
        return {"ids": ids, "kv": _last_head(s.model, 0, 0, c["T"] + c["n_new"] - 1)}
    if s.kind == "step":
        nxt, logits = s.model.decode_step(s.tok, c["ctx"], out=s.logits.array, io=s.io.array)
        return {"next": nxt, "logits": logits}
    if s.kind == "prefill":
        nxt, logits = s.model.prefill(s.prompt, want_logits=True)
        return {"next": nxt, "logits": logits, "kv": _last_head(s.model, 0, 0, c["T"])}
    # the greedy ids, and the K and V row of the last token
    seq = 0
    if s.kind == "loop":
        ids, last = s.model.decode_loop(s.tok, c["ctx"], c["n_new"])[0], c["ctx"] + c["n_new"] - 1
    elif c["ragged"]:
        seq = c["n_seq"] - 1
        ids, last = s.model.decode_batch(s.ids, s.pos), int(s.pos[seq])
    else:
        seq = c["n_seq"] - 1
        ids, last = s.model.decode_batch_loop(s.ids, c["ctx"], c["n_new"])[0], c["ctx"] + c["n_new"] - 1
    return {"ids": ids, "kv": _last_head(s.model, seq, last, 1)}


# ---- what a pass cannot do without --------------------------------------------------------------------------------

PACKED = 0.5625       # bytes of a packed weight: half a byte of code, a sixteenth of a scale byte


def _linear(m):
    """Weights of the layers, weights of the head, bytes of K and V per position."""
    qd, kvd = m["n_heads"] * m["head_dim"], m["n_kv_heads"] * m["head_dim"]
    layer = m["d_model"] * (2 * qd + 2 * kvd + 3 * m["d_ff"])
    return m["n_layers"] * layer, m["vocab"] * m["d_model"], m["n_layers"] * 2 * kvd * 4


def work(case):
    kind = case["kind"]
    if kind in ("quantize", "import", "dequantize"):
        rows, K = case["rows"], case["K"]
        kp = (K + 111) // 112 * 112
        packed = rows * (kp // 7 * 4 + kp // 16)
        if kind == "dequantize":
            return {"bytes": packed + 4 + rows * kp * 4, "flops": rows * kp * 2}
        return {"bytes": rows * K * 4 + packed + rows * (kp // 16) * 4 + 4, "flops": rows * K * 4}
    if kind == "gpt2":
        # every new token reads the weights; the prompt reads them once
        m = dict(GPT2, n_kv_heads=GPT2["n_heads"], head_dim=GPT2["d_model"] // GPT2["n_heads"])
        layers = m["n_layers"] * m["d_model"] * (4 * m["d_model"] + 2 * m["d_ff"])
        head, kv = m["vocab"] * m["d_model"], m["n_layers"] * 2 * m["d_model"] * 4
        T, n = case["T"], case["n_new"]
        attn = sum(T + i for i in range(n))
        return {"bytes": n * (layers + head) * PACKED + kv * attn, "flops": 2 * layers * (T + n - 1) + 2 * head * n + kv * (attn + T * T / 2)}
    m = SHAPES[case["shape"]]
    layers, head, kv = _linear(m)
    per_score = m["n_layers"] * m["n_heads"] * m["head_dim"] * 4      # q.k and p.v of one (query, key) pair in all heads and layers
    if kind == "prefill":
        T = case["T"]
        return {"bytes": (layers + head) * PACKED + T * (kv + m["d_model"] * 4) + m["vocab"] * 4,
                "flops": 2.0 * layers * T + 2.0 * head + per_score * T * (T + 1) / 2}
    n_seq, steps = case.get("n_seq", 1), case.get("n_new", 1)
    if case.get("ragged"):
        cached = n_seq * (case["ctx"] / 2 + 1)         # positions are uniform over [0, ctx]
    else:
        cached = n_seq * (case["ctx"] + (steps + 1) / 2)
    out = m["vocab"] * 4 if kind == "step" else 0
    return {"bytes": steps * ((layers + head) * PACKED + cached * kv + n_seq * m["d_model"] * 4) + out,
            "flops": steps * (2.0 * (layers + head) * n_seq + cached * per_score)}


def tolerance(case):
    if case["kind"] in ("quantize", "import", "dequantize"):
        return "exact"          # codes, scales and their products are defined bit by bit
    # f32 activations and f32 sums in every path, through all layers; greedy ids are equal up to ties
    return {"rel": 2e-5, "max": 2e-4, "differ": 0.01}
