"""The work a user of this package has it do, as measured cases, through the public entry points of `inferred_thoughts_b200.host`.

Four kinds of pass:

  generate  Engine.generate on an empty sequence: a prompt in, greedy tokens out, a host round trip per token.
  prefill   Engine.prefill of one or several prompts of equal length on empty sequences, last token's logits out.
  decode    Engine.decode (one token per sequence in; logits and greedy token out) or Engine.decode_loop (several greedy steps
            without host traffic), on sequences that already hold a prompt. Each pass goes on where the last one stopped.
  ffn       one routed FFN layer of the 35B shape driven op by op through B200Ops, as a host model behind the backend seam
            drives it: rows in from the host, norm, router, top-k, routed and shared experts, weighted combine, rows back.

Shapes are the ones in `inferred_thoughts_b200.configs`; `n_layer` cuts a shape to fewer layers of the same kind. `mode` is the
context's option string. Weights come from the fixed seeds of `configs.SEEDS` (a program loads its model once); the seed handed to
`prepare` makes prompts, tokens and activation rows.
"""
import math
import os
from collections import OrderedDict

import numpy as np

from inferred_thoughts_b200 import configs, host

EXACT = "kv=bf16,exact=1,dense=q8tc"                      # bit-exact arithmetic, the benchmark's headline mode
FAST = "kv=bf16,exact=0,experts=fp4tc,dense=f16tc"        # the tolerance-class kernels, the benchmark's fastest mode
N_CTX = 8192                                              # KV capacity per sequence of the 35B cases (the benchmark's)

SHAPES = {"tiny": configs.TINY, "mid": configs.MID, "odd": configs.ODD, "m35b": configs.M35B}


def listed():
    return [
        # the smallest model, a short chat turn: launches and host round trips are all there is
        dict(name="generate_tiny", kind="generate", shape="tiny", n_layer=4, mode=EXACT, prompt=64, new=32),
        # widths of 24 and 6 blocks, 10 picks, 3 query heads per KV head, a ragged number of rows of several sequences
        dict(name="prefill_odd", kind="prefill", shape="odd", n_layer=4, mode=EXACT, batch=3, prompt=101, rows=512),
        # one user at the terminal, sampling on the host: a token in, the logits out
        dict(name="decode_1", kind="decode", shape="m35b", n_layer=40, mode=EXACT, batch=1, prompt=512, steps=1),
        # the same far into a long conversation, greedy
        dict(name="decode_1_deep", kind="decode", shape="m35b", n_layer=40, mode=EXACT, batch=1, prompt=6500, steps=4),
        # a full batch of users, greedy
        dict(name="decode_32", kind="decode", shape="m35b", n_layer=40, mode=EXACT, batch=32, prompt=128, steps=4),
        # time to first token of an ordinary prompt
        dict(name="prefill_512", kind="prefill", shape="m35b", n_layer=40, mode=EXACT, batch=1, prompt=512, rows=512),
        # a long document, bit-exact
        dict(name="prefill_5548", kind="prefill", shape="m35b", n_layer=40, mode=EXACT, batch=1, prompt=5548, rows=2048),
        # the same through the tolerance-class kernels, on one period of the layer pattern: over 40 layers of random weights a
        # rounding-level difference flips expert picks, and no two correct implementations could be compared
        dict(name="prefill_5548_fast", kind="prefill", shape="m35b", n_layer=4, mode=FAST, batch=1, prompt=5548, rows=2048),
        # the op seam: a decode row, a batch of decode rows, a prompt, and a large pass on the FP4 tensor cores
        dict(name="ffn_1", kind="ffn", mode=EXACT, rows=1),
        dict(name="ffn_32", kind="ffn", mode=EXACT, rows=32),
        dict(name="ffn_500", kind="ffn", mode=EXACT, rows=500),
        dict(name="ffn_2048_fast", kind="ffn", mode=FAST, rows=2048),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any kind, sizes spread over the range between the listed ones."""
    kind = rng.choice(["generate", "prefill", "prefill", "decode", "decode", "ffn"])
    if kind == "generate":
        return dict(kind=kind, shape=rng.choice(["tiny", "mid"]), n_layer=4, mode=EXACT, prompt=_log(rng, 2, 120), new=_log(rng, 4, 40))
    if kind == "prefill":
        which = rng.choice(["small", "exact", "fast"])
        if which == "small":
            return dict(kind=kind, shape=rng.choice(["odd", "mid"]), n_layer=4, mode=EXACT, batch=rng.randint(1, 6), prompt=_log(rng, 5, 300), rows=512)
        if which == "exact":
            return dict(kind=kind, shape="m35b", n_layer=40, mode=EXACT, batch=1, prompt=_log(rng, 20, 3000), rows=rng.choice([512, 2048]))
        return dict(kind=kind, shape="m35b", n_layer=4, mode=FAST, batch=1, prompt=_log(rng, 100, 5548), rows=2048)
    if kind == "decode":
        batch = rng.choice([1, _log(rng, 2, 32)])
        return dict(kind=kind, shape="m35b", n_layer=40, mode=EXACT, batch=batch, prompt=_log(rng, 16, 5000) if batch == 1 else _log(rng, 16, 200),
                    steps=rng.choice([1, 2, 4]))
    return dict(kind=kind, mode=rng.choice([EXACT, FAST]), rows=_log(rng, 1, 2048))


# ---- what a program has in hand -----------------------------------------------------------------------------------
_kept = OrderedDict()      # contexts with their model or layer weights: the two most recent ones


def _keep(key, make):
    if key not in _kept:
        while len(_kept) >= 2:
            _kept.popitem(last=False)
        _kept[key] = make()
    _kept.move_to_end(key)
    return _kept[key]


def _model(case):
    dims = configs.with_layers(SHAPES[case["shape"]], case["n_layer"])

    def make():
        ops = host.B200Ops(0, case["mode"])
        model = host.Model(ops, host.ModelDims(**dims))
        model.synth(configs.SEEDS[case["shape"]])
        return model
    return dims, _keep((case["shape"], case["n_layer"], case["mode"]), make)


def _engine(model, n_ctx, batch, rows):
    """An engine whose many-row passes take `rows` rows (the library reads ITB_ROWS when an engine is made)."""
    before = os.environ.get("ITB_ROWS")
    os.environ["ITB_ROWS"] = str(rows)
    try:
        return host.Engine(model, n_ctx, batch)
    finally:
        if before is None:
            del os.environ["ITB_ROWS"]
        else:
            os.environ["ITB_ROWS"] = before


class _Layer:
    """A context and one routed FFN layer of the 35B shape in the file's block layouts: NVFP4 expert stacks with a second scale per
    expert, Q8_0 shared expert, F32 router and gate. Valid blocks with the magnitudes of N(0, 0.02) weights."""

    def __init__(self, mode):
        d = configs.M35B
        H, ff, E, sff = d["n_embd"], d["expert_ff"], d["n_expert"], d["shared_ff"]
        rng = np.random.default_rng(configs.SEEDS["m35b"])
        self.ops = host.B200Ops(0, mode)

        def fp4(n_in, n_out):
            b = np.frombuffer(rng.bytes(E * n_in * n_out // 64 * 36), np.uint8).reshape(-1, 36).copy()
            b[:, :4] = 0x28 + (b[:, :4] & 0x0f)
            return host.Experts(b.reshape(-1), host.NVFP4, n_in, n_out, E, (0.004 + 0.004 * rng.random(E)).astype(np.float32))

        def q8(n_in, n_out):
            b = np.frombuffer(rng.bytes(n_in * n_out // 32 * 34), np.uint8).reshape(-1, 34).copy()
            b[:, :2] = (0.0002 + 0.0002 * rng.random(len(b))).astype(np.float16).view(np.uint8).reshape(-1, 2)
            return host.Weights(b.reshape(-1), host.Q8_0, n_in, n_out)

        def f32(n_in, n_out):
            return host.Weights((0.02 * rng.standard_normal(n_in * n_out)).astype(np.float32), host.F32, n_in, n_out)
        self.norm = (1.0 + 0.02 * rng.standard_normal(H)).astype(np.float32)
        self.router, self.gate_logit = f32(H, E), f32(H, 1)
        self.gate, self.up, self.down = fp4(H, ff), fp4(H, ff), fp4(ff, H)
        self.sh_gate, self.sh_up, self.sh_down = q8(H, sff), q8(H, sff), q8(sff, H)


class _State:
    pass


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    s = _State()
    s.case = dict(case)
    if case["kind"] == "ffn":
        d = configs.M35B
        H, ff, E, K, sff, T = d["n_embd"], d["expert_ff"], d["n_expert"], d["n_expert_used"], d["shared_ff"], case["rows"]
        s.layer = _keep(("ffn", case["mode"]), lambda: _Layer(case["mode"]))
        s.x = rng.standard_normal(T * H).astype(np.float32)
        zeros = lambda n: np.zeros(n, np.float32)  # noqa: E731
        s.normed, s.router, s.logit = zeros(T * H), zeros(T * E), zeros(T)
        s.h, s.scratch, s.o = zeros(T * K * ff), zeros(T * K * ff), zeros(T * K * H)
        s.sg, s.su, s.sh, s.out = zeros(T * sff), zeros(T * sff), zeros(T * H), zeros(T * H)
        return s
    dims, model = _model(case)
    vocab = dims["n_vocab"]
    if case["kind"] == "generate":
        s.eng = _engine(model, case["prompt"] + case["new"] + 1, 1, 512)
        s.prompt = rng.integers(0, vocab, case["prompt"]).astype(np.uint32)
    elif case["kind"] == "prefill":
        n_ctx = N_CTX if case["shape"] == "m35b" else 512
        s.eng = _engine(model, n_ctx, case["batch"], case["rows"])
        s.prompt = rng.integers(0, vocab, (case["batch"], case["prompt"])).astype(np.uint32)
    else:
        s.eng = _engine(model, N_CTX, case["batch"], 512)
        s.eng.prefill(rng.integers(0, vocab, (case["batch"], case["prompt"])).astype(np.uint32), want_logits=False)
        s.token = rng.integers(0, vocab, case["batch"]).astype(np.uint32)
    return s


# ---- the passes ---------------------------------------------------------------------------------------------------
def run(s):
    return {"generate": _generate, "prefill": _prefill, "decode": _decode, "ffn": _ffn}[s.case["kind"]](s)


def _generate(s):
    s.eng.reset()
    return {"tokens": s.eng.generate(s.prompt, s.case["new"])}


def _prefill(s):
    s.eng.reset()
    return {"logits": s.eng.prefill(s.prompt)}


def _decode(s):
    steps = s.case["steps"]
    if s.eng.pos() + steps > N_CTX:      # the conversation is full: begin the next one
        s.eng.reset()
    if steps == 1:
        logits, s.token = s.eng.decode(s.token)
        return {"logits": logits, "next": s.token}
    tokens = s.eng.decode_loop(s.token, steps)
    s.token = tokens[-1].copy()
    return {"tokens": tokens}


def _ffn(s):
    d, w = configs.M35B, s.layer
    H, E, K = d["n_embd"], d["n_expert"], d["n_expert_used"]
    ops = w.ops
    ops.begin_pass(s.case["rows"])
    ops.rms_norm(s.x, w.norm, d["rms_eps"], s.normed)
    ops.matmul_pair(w.router, w.gate_logit, s.normed, s.router, s.logit)
    ops.softmax(s.router, E)
    route = ops.route(s.router, E, K)
    ops.moe_glu(w.gate, w.up, route, s.normed, s.h, s.scratch)
    ops.matmul_experts(w.down, route, s.h, s.o)
    ops.matmul_pair(w.sh_gate, w.sh_up, s.normed, s.sg, s.su)
    ops.silu_mul(s.sg, s.su)
    ops.matmul(w.sh_down, s.sg, s.sh)
    ops.moe_finish(s.out, 0, H, s.o, route, s.sh, s.logit, 0)
    ops.host_needs(s.out)
    ops.end_pass()
    ops.check()
    return {"out": s.out}


# ---- what a pass cannot do without --------------------------------------------------------------------------------
def _q8(n_in, n_out):
    return n_in * n_out / 32 * 34


def _fp4(n_in, n_out):
    return n_in * n_out / 64 * 36


def _distinct(E, pairs):
    """Expected number of distinct experts among that many uniform picks."""
    return E * (1.0 - (1.0 - 1.0 / E) ** pairs)


def _pass_work(d, n_seq, n_tok, pos, heads):
    """n_tok tokens of each of n_seq sequences that hold `pos` tokens already; logits for `heads` rows. Weights once each (routed
    experts: those hit), recurrent state read and written, KV read once per sequence and written once, embedding rows."""
    H, E, K, ff, sff = d["n_embd"], d["n_expert"], d["n_expert_used"], d["expert_ff"], d["shared_ff"]
    key, vd, sk, n_v = d["ssm_d_state"] * d["ssm_n_group"], d["ssm_d_inner"], d["ssm_d_state"], d["ssm_dt_rank"]
    cd, qd, kvd = 2 * key + vd, d["head_dim"] * d["n_head"], d["head_dim"] * d["n_head_kv"]
    rows = n_seq * n_tok
    ffn_b = _distinct(E, rows * K) * 3 * _fp4(H, ff) + 4 * H * (E + 1) + 3 * _q8(H, sff)
    ffn_f = 2 * rows * (3 * K * H * ff + H * (E + 1) + 3 * H * sff)
    gdn_b = _q8(H, cd) + _q8(H, vd) + _q8(vd, H) + 8 * H * n_v + 4 * cd * d["ssm_d_conv"] + n_seq * 8 * (n_v * sk * sk + (d["ssm_d_conv"] - 1) * cd)
    gdn_f = 2 * rows * (H * cd + 2 * H * vd + 2 * H * n_v + cd * d["ssm_d_conv"] + 3 * n_v * sk * sk)
    att_b = _q8(H, 2 * qd) + 2 * _q8(H, kvd) + _q8(qd, H) + n_seq * 4 * kvd * (pos + n_tok)
    att_f = 2 * rows * (3 * H * qd + 2 * H * kvd + 2 * qd * (pos + (n_tok + 1) / 2))
    n_att = d["n_layer"] // d["full_attention_interval"]
    n_rec = d["n_layer"] - n_att
    return (d["n_layer"] * ffn_b + n_rec * gdn_b + n_att * att_b + _q8(H, d["n_vocab"]) + 4 * (rows * H + heads * d["n_vocab"]),
            d["n_layer"] * ffn_f + n_rec * gdn_f + n_att * att_f + 2 * heads * H * d["n_vocab"])


def work(case):
    if case["kind"] == "ffn":
        d, T = configs.M35B, case["rows"]
        H, E, K, ff, sff = d["n_embd"], d["n_expert"], d["n_expert_used"], d["expert_ff"], d["shared_ff"]
        return {"bytes": _distinct(E, T * K) * 3 * _fp4(H, ff) + 4 * H * (E + 1) + 3 * _q8(H, sff) + 8 * T * H,
                "flops": 2 * T * (3 * K * H * ff + H * (E + 1) + 3 * H * sff)}
    d = configs.with_layers(SHAPES[case["shape"]], case["n_layer"])
    if case["kind"] == "generate":
        b, f = _pass_work(d, 1, case["prompt"], 0, 1)
        for i in range(case["new"] - 1):
            sb, sf = _pass_work(d, 1, 1, case["prompt"] + i, 1)
            b, f = b + sb, f + sf
        return {"bytes": b, "flops": f}
    if case["kind"] == "prefill":
        b, f = _pass_work(d, case["batch"], case["prompt"], 0, case["batch"])
    else:
        b, f = _pass_work(d, case["batch"], 1, case["prompt"], case["batch"])
        b, f = b * case["steps"], f * case["steps"]
    return {"bytes": b, "flops": f}


def tolerance(case):
    """exact=1 promises the CPU path's bits. The tolerance-class mode multiplies FP4, f16 and bf16 operands, so results agree to
    what those types give."""
    return "exact" if case["mode"] == EXACT else {"rel": 1e-2}
