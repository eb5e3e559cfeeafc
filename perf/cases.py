"""The work this package is used for, as measurable cases.

A case is one pass through the prepared operators of ``tuiskollm_b200`` the way a serving program
calls them: the decode and prefill halves of a transformer layer, the MLP in both weight formats,
and the head that turns hidden rows into tokens.  ``rows`` is the number of tokens in the call.

``graph`` says how a decode step is issued: captured once and replayed (what an engine with a fixed
batch does), or operator by operator (what a Python program does, and what prefill does anyway,
since its row count changes from call to call).

Shapes are the model's: hidden 5120, MLP 17408, 248320 tokens; FP8 projections of 8192 and 12288
rows (14336 and 16384 with the fused gate and value rows).
"""
from __future__ import annotations

import torch

import tuiskollm_b200 as tk
from tuiskollm_b200 import ops, synth

HIDDEN = synth.HIDDEN
INTER = synth.INTERMEDIATE
VALUE_WIDTH = 6144        # 48 value heads of 128: the GDN output projection's reduction
CONV_CHANNELS = 10240
CONTROL_ROWS = 96
STATE_WORDS = 48 * 128 * 128

# calibration constants of the NVFP4 activation quantisers: ~N(0, 1) rows, SwiGLU outputs
HIDDEN_DIVISOR = 448.0 * 6.0 / 6.0
MID_DIVISOR = 448.0 * 6.0 / 8.0


def listed():
    return [
        # The smallest call: residual add, RMSNorm and E4M3 quantisation of one token.
        {"name": "norm_1", "kind": "norm", "rows": 1, "nvfp4": False, "graph": False},
        # Into the attention of one decoded token, called operator by operator.
        {"name": "attention_in_1", "kind": "attention_in", "rows": 1, "out_rows": 8192, "graph": False},
        # Into the attention of a long, odd-sized prompt (fused query and gate rows).
        {"name": "attention_in_1777", "kind": "attention_in", "rows": 1777, "out_rows": 14336, "graph": False},
        # A gated-delta-net layer for one request, as an engine replays it.
        {"name": "gdn_layer_1", "kind": "gdn_layer", "rows": 1, "graph": True},
        # The same layer for an odd batch, operator by operator.
        {"name": "gdn_layer_7", "kind": "gdn_layer", "rows": 7, "graph": False},
        # The quantized projections of a layer, one decoded token: the decode headline.
        {"name": "slice_1", "kind": "slice", "rows": 1, "graph": True},
        # The same for 512 tokens: a large decode batch or a prompt chunk, the prefill headline.
        {"name": "slice_512", "kind": "slice", "rows": 512, "graph": False},
        # NVFP4 MLP between decode and prefill, a ragged token count.
        {"name": "nvfp4_mlp_100", "kind": "nvfp4_mlp", "rows": 100, "graph": False},
        # NVFP4 MLP of a full prefill chunk: the largest contraction.
        {"name": "nvfp4_mlp_2048", "kind": "nvfp4_mlp", "rows": 2048, "graph": False},
        # MLP with dense FP8 weights, a short odd-sized prompt.
        {"name": "fp8_mlp_301", "kind": "fp8_mlp", "rows": 301, "graph": False},
        # Greedy decoding of one request: fp32 logits and the argmax of the whole vocabulary.
        {"name": "greedy_head_1", "kind": "greedy_head", "rows": 1, "vocab": synth.VOCAB, "graph": True},
        # Sampled decoding of eight requests: LM head, then top-k / top-p on the device.
        {"name": "sampled_head_8", "kind": "sampled_head", "rows": 8, "vocab": synth.VOCAB, "graph": False},
    ]


def _rows(rng, low, high):
    """A row count spread over the logarithm of [low, high]."""
    return max(low, min(high, int(round(low * (high / low) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["norm", "attention_in", "attention_in", "gdn_layer", "slice", "nvfp4_mlp", "nvfp4_mlp",
                       "fp8_mlp", "greedy_head", "sampled_head"])
    case = {"kind": kind}
    if kind == "norm":
        case.update(rows=_rows(rng, 1, 2048), nvfp4=rng.random() < 0.5)
    elif kind == "attention_in":
        case.update(rows=_rows(rng, 1, 2048), out_rows=rng.choice([8192, 12288, 14336, 16384]))
    elif kind == "gdn_layer":
        case.update(rows=rng.randint(1, 8))
    elif kind == "slice":
        case.update(rows=_rows(rng, 1, 1024))
    elif kind in ("nvfp4_mlp", "fp8_mlp"):
        case.update(rows=_rows(rng, 1, 2048 if kind == "nvfp4_mlp" else 1024))
    else:
        # the whole vocabulary or what one of several devices holds of it
        vocab = 16 * rng.randrange(synth.VOCAB // 128, synth.VOCAB // 16)
        case.update(rows=_rows(rng, 1, 32) if kind == "greedy_head" else rng.randint(1, 8), vocab=vocab)
    case["graph"] = case["rows"] <= 32 and rng.random() < 0.5
    return case


# ------------------------------------------------------------------------------- planes

class _Planes:
    """Seeded planes; every tensor has a random stream of its own."""

    def __init__(self, seed):
        self.seed, self.stream = seed, 0

    def _next(self):
        self.stream += 1
        return self.stream

    def bf16(self, *shape, std=1.0):
        return synth.torch_normal_bf16(self.seed, self._next(), shape, "cuda", std=std)

    def fp8(self, rows, k):
        return synth.torch_fp8_weights(self.seed, self._next(), rows, k, "cuda")

    def nvfp4(self, rows, k):
        return synth.torch_nvfp4_weights(self.seed, self._next(), rows, k, "cuda")

    def f32(self, *shape, std=1.0):
        g = torch.Generator(device="cuda").manual_seed((self.seed * 1000003 + self._next()) & 0x7FFFFFFFFFFFFFFF)
        return torch.randn(shape, generator=g, device="cuda") * std


def _bf16_out(*shape):
    return torch.zeros(shape, dtype=torch.bfloat16, device="cuda")


def _e4m3_planes(rows, k):
    return (torch.zeros((rows, k), dtype=torch.uint8, device="cuda"),
            torch.zeros((rows,), dtype=torch.float32, device="cuda"))


def _nvfp4_planes(rows, k):
    return (torch.zeros((rows, k // 2), dtype=torch.uint8, device="cuda"),
            torch.zeros((ops.nvfp4_scale_plane_bytes(rows, k),), dtype=torch.uint8, device="cuda"))


# ------------------------------------------------------------------------------ the paths
# Each builder returns (step, outputs, mutable): the call sequence of one pass, the planes it
# leaves, and the planes a pass changes that the next one reads.

def _norm_step(ctx, p, rows, nvfp4):
    """The fused producer in front of every projection."""
    x, branch = p.bf16(rows, HIDDEN), p.bf16(rows, HIDDEN)
    weight = p.bf16(HIDDEN, std=0.1)
    residual, normed = _bf16_out(rows, HIDDEN), _bf16_out(rows, HIDDEN)
    codes, scales = _e4m3_planes(rows, HIDDEN)
    op = tk.ResidualNormOp(ctx)
    if nvfp4:
        c4, s4 = _nvfp4_planes(rows, HIDDEN)

        def step():
            op.launch_quantize_nvfp4(None, rows, x, branch, weight, residual, normed, codes, scales,
                                     HIDDEN_DIVISOR, c4, s4)

        return step, {"residual": residual, "normed": normed, "codes": codes, "scales": scales,
                      "codes4": c4, "scales4": s4}

    def step():
        op.launch_quantize(None, rows, x, branch, weight, residual, normed, codes, scales)

    return step, {"residual": residual, "normed": normed, "codes": codes, "scales": scales}


def _norm(ctx, p, case):
    step, out = _norm_step(ctx, p, case["rows"], case["nvfp4"])
    return step, out, []


def _attention_in(ctx, p, case):
    rows, n = case["rows"], case["out_rows"]
    norm, made = _norm_step(ctx, p, rows, False)
    w, ws = p.fp8(n, HIDDEN)
    ctx.register_plane(w)
    out = _bf16_out(rows, n)
    op = tk.FullAttentionQkvOp(ctx, n)

    def step():
        norm()
        op.launch(None, rows, None, made["codes"], made["scales"], w, ws, out)

    return step, {"residual": made["residual"], "projected": out}, []


def _gdn_layer(ctx, p, case):
    rows = case["rows"]
    norm, made = _norm_step(ctx, p, rows, False)
    w_in, ws_in = p.fp8(synth.GDN_ROWS_REF, HIDDEN)
    w_out, ws_out = p.fp8(HIDDEN, VALUE_WIDTH)
    for w in (w_in, w_out):
        ctx.register_plane(w)
    control = p.bf16(CONTROL_ROWS, HIDDEN, std=0.02)
    a_log, dt_bias = p.bf16(48), p.bf16(48)
    conv_w = p.bf16(CONV_CHANNELS, 4, std=0.5)
    norm_w = p.bf16(128)
    slots = 8
    order = torch.randperm(slots, generator=torch.Generator().manual_seed(p.seed))[:rows]
    slot_of = order.to(torch.int32).cuda()
    history = p.bf16(slots, CONV_CHANNELS, 3)
    state = p.f32(slots, 48, 128, 128, std=0.05)
    projected, convolved = _bf16_out(rows, synth.GDN_ROWS_REF), _bf16_out(rows, CONV_CHANNELS)
    decay = torch.zeros((rows, 48), dtype=torch.float32, device="cuda")
    beta = torch.zeros_like(decay)
    mixed, out = _bf16_out(rows, VALUE_WIDTH), _bf16_out(rows, HIDDEN)
    codes, scales = _e4m3_planes(rows, VALUE_WIDTH)
    in_op = tk.GdnInputProjectionOp(ctx, synth.GDN_ROWS_REF)
    prepare_op, recurrence_op = tk.GdnPrepareOp(ctx), tk.GdnRecurrenceOp(ctx)
    out_op = tk.GdnOutputProjectionOp(ctx, VALUE_WIDTH)

    def step():
        norm()
        in_op.launch(None, rows, None, made["codes"], made["scales"], w_in, ws_in, projected)
        prepare_op.launch(None, rows, made["normed"], control, a_log, dt_bias, projected, conv_w, slot_of,
                          history, decay, beta, convolved)
        recurrence_op.launch(None, rows, convolved, projected, decay, beta, norm_w, slot_of, state, mixed)
        out_op.launch(None, rows, mixed, codes, scales, w_out, ws_out, out)

    return step, {"residual": made["residual"], "history": history, "state": state, "out": out}, [history, state]


class _Nvfp4Mlp:
    def __init__(self, ctx, p, rows):
        self.rows = rows
        self.gu = p.nvfp4(2 * INTER, HIDDEN)
        self.dn = p.nvfp4(HIDDEN, INTER)
        for plane in (self.gu[0], self.dn[0]):
            ctx.register_plane(plane)
        self.mid, self.out = _bf16_out(rows, INTER), _bf16_out(rows, HIDDEN)
        self.mid_codes, self.mid_scales = _nvfp4_planes(rows, INTER)
        self.up_op, self.down_op = tk.Nvfp4SwiGluOp(ctx), tk.Nvfp4DownOp(ctx)

    def step(self, codes, scales):
        self.up_op.launch_quantize(None, self.rows, None, *self.gu, self.mid, activation_codes=codes,
                                   activation_scales=scales, input_global_divisor=HIDDEN_DIVISOR,
                                   output_global_divisor=MID_DIVISOR, output_codes=self.mid_codes,
                                   output_scales=self.mid_scales)
        self.down_op.launch(None, self.rows, None, *self.dn, self.out, activation_codes=self.mid_codes,
                            activation_scales=self.mid_scales, input_global_divisor=MID_DIVISOR)


def _nvfp4_mlp(ctx, p, case):
    rows = case["rows"]
    norm, made = _norm_step(ctx, p, rows, True)
    mlp = _Nvfp4Mlp(ctx, p, rows)

    def step():
        norm()
        mlp.step(made["codes4"], made["scales4"])

    return step, {"residual": made["residual"], "mid": mlp.mid, "out": mlp.out}, []


def _slice(ctx, p, case):
    rows = case["rows"]
    norm, made = _norm_step(ctx, p, rows, True)
    w_q, ws_q = p.fp8(synth.QKV_ROWS, HIDDEN)
    w_g, ws_g = p.fp8(synth.GDN_ROWS, HIDDEN)
    for w in (w_q, w_g):
        ctx.register_plane(w)
    mlp = _Nvfp4Mlp(ctx, p, rows)
    qkv, gdn = _bf16_out(rows, synth.QKV_ROWS), _bf16_out(rows, synth.GDN_ROWS)
    qkv_op = tk.FullAttentionQkvOp(ctx, synth.QKV_ROWS)
    gdn_op = tk.GdnInputProjectionOp(ctx, synth.GDN_ROWS)

    def step():
        norm()
        qkv_op.launch(None, rows, None, made["codes"], made["scales"], w_q, ws_q, qkv)
        gdn_op.launch(None, rows, None, made["codes"], made["scales"], w_g, ws_g, gdn)
        mlp.step(made["codes4"], made["scales4"])

    return step, {"residual": made["residual"], "qkv": qkv, "gdn": gdn, "out": mlp.out}, []


def _fp8_mlp(ctx, p, case):
    rows = case["rows"]
    norm, made = _norm_step(ctx, p, rows, False)
    gu, gus = p.fp8(2 * INTER, HIDDEN)
    dn, dns = p.fp8(HIDDEN, INTER)
    for w in (gu, dn):
        ctx.register_plane(w)
    mid, out = _bf16_out(rows, INTER), _bf16_out(rows, HIDDEN)
    codes, scales = _e4m3_planes(rows, INTER)
    up_op, down_op = tk.Fp8SwiGluOp(ctx), tk.Fp8DownOp(ctx)

    def step():
        norm()
        up_op.launch(None, rows, None, made["codes"], made["scales"], gu, gus, mid)
        down_op.launch(None, rows, mid, codes, scales, dn, dns, out)

    return step, {"residual": made["residual"], "mid": mid, "out": out}, []


def _head(ctx, p, case, sampled):
    rows, vocab = case["rows"], case["vocab"]
    norm, made = _norm_step(ctx, p, rows, False)
    w, ws = p.fp8(vocab, HIDDEN)
    ctx.register_plane(w)
    logits = _bf16_out(rows, vocab)
    op = tk.LmHeadOp(ctx, vocab)
    if sampled:
        options = [tk.SamplingOptions.greedy() if i % 4 == 3 else
                   tk.SamplingOptions(temperature=0.7 + 0.1 * i, top_p=0.95, top_k=20, seed=p.seed + i)
                   for i in range(rows)]
        sampler = tk.Sampler(ctx, vocab, options, [(1, 2)] * rows)

        def step():
            norm()
            op.launch(None, rows, None, made["codes"], made["scales"], w, ws, logits)
            sampler.sample(None, logits)

        return step, {"logits": logits, "decisions": sampler.decisions, "rng": sampler.rng_state}, [sampler.rng_state]

    logits_f32 = torch.zeros((rows, vocab), dtype=torch.float32, device="cuda")
    scratch = torch.zeros((rows,), dtype=torch.int64, device="cuda")
    pairs = torch.zeros((rows, 2), dtype=torch.int32, device="cuda")

    def step():
        norm()
        op.launch(None, rows, None, made["codes"], made["scales"], w, ws, logits, logits_f32, scratch, pairs)

    return step, {"logits": logits, "logits_f32": logits_f32, "value": pairs.view(torch.float32)[:, 0],
                  "token": pairs[:, 1]}, []


_BUILDERS = {
    "norm": _norm, "attention_in": _attention_in, "gdn_layer": _gdn_layer, "slice": _slice,
    "nvfp4_mlp": _nvfp4_mlp, "fp8_mlp": _fp8_mlp,
    "greedy_head": lambda ctx, p, case: _head(ctx, p, case, False),
    "sampled_head": lambda ctx, p, case: _head(ctx, p, case, True),
}


def prepare(case, seed):
    ctx = tk.Context(device=torch.cuda.current_device())
    step, outputs, mutable = _BUILDERS[case["kind"]](ctx, _Planes(seed), case)
    call = step
    graph = None
    if case["graph"]:
        kept = [t.clone() for t in mutable]
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            step()
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            step()
        for t, k in zip(mutable, kept):
            t.copy_(k)
        call = graph.replay
    return {"call": call, "outputs": outputs, "context": ctx, "step": step, "graph": graph}


def run(state):
    state["call"]()
    return state["outputs"]


# ----------------------------------------------------------------- what a pass cannot avoid

def work(case):
    rows, kind = case["rows"], case["kind"]
    # residual and branch in, residual out, norm weight
    nbytes, flops = rows * 6.0 * HIDDEN + 2.0 * HIDDEN, 0.0

    def fp8(n, k, out_bytes):
        nonlocal nbytes, flops
        nbytes += n * k + 2 * n + out_bytes
        flops += 2.0 * rows * n * k

    def nvfp4(n, k, out_bytes):
        nonlocal nbytes, flops
        nbytes += n * k * 9 / 16 + out_bytes
        flops += 2.0 * rows * n * k

    if kind == "norm":
        nbytes += rows * (3.0 * HIDDEN + 4) + (rows * HIDDEN * 9 / 16 if case["nvfp4"] else 0)
    elif kind == "attention_in":
        fp8(case["out_rows"], HIDDEN, 2 * rows * case["out_rows"])
    elif kind == "gdn_layer":
        fp8(synth.GDN_ROWS_REF, HIDDEN, 0)
        fp8(HIDDEN, VALUE_WIDTH, 2 * rows * HIDDEN)
        nbytes += 2 * CONTROL_ROWS * HIDDEN + 8 * CONV_CHANNELS + rows * (8 * STATE_WORDS + 12 * CONV_CHANNELS)
        flops += rows * (2.0 * CONTROL_ROWS * HIDDEN + 8.0 * CONV_CHANNELS + 7.0 * STATE_WORDS)
    elif kind == "slice":
        fp8(synth.QKV_ROWS, HIDDEN, 2 * rows * synth.QKV_ROWS)
        fp8(synth.GDN_ROWS, HIDDEN, 2 * rows * synth.GDN_ROWS)
        nvfp4(2 * INTER, HIDDEN, 2 * rows * INTER)
        nvfp4(HIDDEN, INTER, 2 * rows * HIDDEN)
    elif kind == "nvfp4_mlp":
        nvfp4(2 * INTER, HIDDEN, 2 * rows * INTER)
        nvfp4(HIDDEN, INTER, 2 * rows * HIDDEN)
    elif kind == "fp8_mlp":
        fp8(2 * INTER, HIDDEN, 2 * rows * INTER)
        fp8(HIDDEN, INTER, 2 * rows * HIDDEN)
    else:
        fp8(case["vocab"], HIDDEN, (6 if kind == "greedy_head" else 2) * rows * case["vocab"])
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """BF16 results of contractions whose operands were rounded to 8 or 4 bits: another correct
    order of the fp32 sums moves single results by one BF16 step (2^-8) and, through the second
    quantiser of an MLP, single codes.  Codes and scales of the fused producer follow its BF16
    row, so a code differs only where that row's last bit does."""
    if case["kind"] == "norm":
        return {"rel": 2e-3, "max": 0.3, "differ": 2e-3}
    if case["kind"] in ("greedy_head", "sampled_head"):
        return {"rel": 4e-3, "max": 0.05, "differ": 0.0}
    return {"rel": 1e-2, "max": 0.3}
