"""What the speed of this framework is measured on: calls of its public entry points as programs make them.

A case is one pass of one of four callers:

* ``step``: one decoding step, a batch of sequences with one new token each, state in and state out;
* ``prefill``: the forward alone over prompts, with the final states that decoding goes on from;
* ``train``: forward and backward of the op (``ops.linear_attention``; ``layers.mamba2_ssd`` for the kind ``ssd``);
* ``layer``: forward and backward of a Gated DeltaNet mixer between its projections (short convolutions of q, k and v,
  gate activations, the op, gated RMS norm).

``docs`` says how documents share the tokens: ``none`` (one per batch row), ``segments`` (``segment_ids`` that restart
the state inside a row) or ``rows`` (``cu_seqlens``, ``seqs`` of them with a state each).
"""

import math
import random

import torch

from jax_linear_attention_b200 import ops
from jax_linear_attention_b200.layers import gate_prologue, gated_rms_norm, mamba2_ssd, short_conv

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}


def _case(name, mode, kind, B, T, H, K, V, *, Hk=None, dtype="bf16", docs="none", lo=0, hi=0, seqs=0, l2norm=False,
          state=False):
    """``lo``, ``hi``: shortest and longest document of ``segments``; ``state``: an initial state comes in."""
    c = dict(mode=mode, kind=kind, B=B, T=T, H=H, Hk=Hk or H, K=K, V=V, dtype=dtype, docs=docs, lo=lo, hi=hi, seqs=seqs,
             l2norm=l2norm, state=state)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # serving: every token that is generated is one of these calls per layer
        _case("gdn_step", "step", "gated_deltanet", 64, 1, 16, 128, 128, l2norm=True, state=True),
        _case("ssd_step", "step", "ssd", 8, 1, 64, 128, 64, Hk=1, state=True),
        # serving: prompts of odd lengths packed into one call, each going on from a state of its own
        _case("gdn_prefill_packed", "prefill", "gated_deltanet", 1, 5003, 16, 128, 128, Hk=8, docs="rows", seqs=9,
              l2norm=True, state=True),
        # serving: one fresh prompt, per-channel gates
        _case("kda_prefill", "prefill", "kda", 1, 4100, 16, 128, 128),
        # the headline training workload: packed documents, heads of 128
        _case("gdn_train", "train", "gated_deltanet", 8, 2048, 16, 128, 128, docs="segments", lo=64, hi=2048),
        # a small model in float16: heads of 64, grouped keys, a ragged length
        _case("gdn_train_d64", "train", "gated_deltanet", 3, 1000, 8, 64, 64, Hk=4, dtype="f16", docs="segments", lo=64,
              hi=1000, l2norm=True),
        # the usual Gated DeltaNet layout: values twice as wide as keys
        _case("gdn_train_wide", "train", "gated_deltanet", 8, 2048, 16, 128, 256, docs="segments", lo=64, hi=2048),
        # per-channel gates (Kimi Delta Attention)
        _case("kda_train", "train", "kda", 4, 4096, 16, 128, 128, docs="segments", lo=128, hi=4096),
        # Mamba-2's SSD scan: one B, C group for all heads, skip term
        _case("ssd_train", "train", "ssd", 8, 2048, 64, 128, 64, Hk=1),
        # everything between the projections of one Gated DeltaNet layer
        _case("gdn_layer_train", "layer", "gated_deltanet", 4, 2048, 16, 128, 128, docs="segments", lo=64, hi=2048),
        # the float32 configuration (numerics work, gradient checks)
        _case("gdn_f32_train", "train", "gated_deltanet", 1, 512, 4, 64, 64, dtype="f32"),
        # long context: one row, long documents
        _case("gdn_long_train", "train", "gated_deltanet", 1, 131072, 16, 128, 128, docs="segments", lo=4096, hi=131072),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _length(rng, lo, hi):
    """A length, spread over its logarithm; every other one rounded to a whole number of 64 tokens."""
    n = _log_int(rng, lo, hi)
    return n if rng.random() < 0.5 else max(lo, n // 64 * 64)


def _fit(tokens, batch):
    """The longest length that ``batch`` rows may have in ``tokens`` tokens."""
    return max(64, tokens // batch)


def draw(rng):
    family = rng.choice(["step", "step_ssd", "prefill", "prefill_rows", "train", "train_d64", "train_wide", "train_channel",
                         "train_ssd", "layer", "f32", "long"])
    dtype = rng.choice(["bf16", "bf16", "f16"])
    heads = rng.choice([4, 8, 12, 16])
    if family == "step":
        kind = rng.choice(["gated_deltanet", "gated_deltanet", "kda", "gdn2", "deltanet"])
        groups = 1 if kind == "gdn2" else rng.choice([1, 1, 2])
        return _case(None, "step", kind, _log_int(rng, 1, 128), 1, heads, 128, 128, Hk=heads // groups, dtype=dtype,
                     l2norm=rng.random() < 0.5, state=True)
    if family == "step_ssd":
        return _case(None, "step", "ssd", _log_int(rng, 1, 64), 1, rng.choice([24, 32, 64]), 128, 64, Hk=rng.choice([1, 8]),
                     dtype=dtype, state=True)
    if family == "prefill":
        kind = rng.choice(["gated_deltanet", "kda", "simple_gla"])
        batch = rng.choice([1, 2, 4])
        return _case(None, "prefill", kind, batch, _length(rng, 64, 8192 // batch), heads, 128, 128, dtype=dtype,
                     l2norm=kind != "simple_gla" and rng.random() < 0.5, state=rng.random() < 0.5)
    if family == "prefill_rows":
        seqs = _log_int(rng, 2, 32)
        kind = rng.choice(["gated_deltanet", "gated_deltanet", "kda"])
        return _case(None, "prefill", kind, 1, _log_int(rng, 8 * seqs, 16384), heads, 128, 128, Hk=heads // rng.choice([1, 2]),
                     dtype=dtype, docs="rows", seqs=seqs, l2norm=rng.random() < 0.5, state=rng.random() < 0.5)
    if family == "train":
        batch, kind = rng.choice([1, 2, 4, 8]), rng.choice(["gated_deltanet", "gated_deltanet", "deltanet", "simple_gla"])
        n = _length(rng, 64, _fit(16384, batch))
        return _case(None, "train", kind, batch, n, heads, 128, 128, Hk=heads // rng.choice([1, 1, 2]), dtype=dtype,
                     docs=rng.choice(["none", "segments"]), lo=min(64, n), hi=n,
                     l2norm=kind != "simple_gla" and rng.random() < 0.5, state=rng.random() < 0.25)
    if family == "train_d64":
        batch = rng.choice([1, 2, 3, 8])
        n = _length(rng, 64, _fit(16384, batch))
        k, v = rng.choice([(64, 64), (64, 64), (64, 128), (128, 64)])
        return _case(None, "train", "gated_deltanet", batch, n, heads, k, v, Hk=heads // rng.choice([1, 2]), dtype=dtype,
                     docs=rng.choice(["none", "segments"]), lo=min(64, n), hi=n, l2norm=rng.random() < 0.5)
    if family == "train_wide":
        batch = rng.choice([1, 2, 4, 8])
        n = _length(rng, 64, _fit(16384, batch))
        return _case(None, "train", "gated_deltanet", batch, n, rng.choice([4, 8, 16]), 128, rng.choice([256, 256, 512]),
                     dtype=dtype, docs=rng.choice(["none", "segments"]), lo=min(64, n), hi=n)
    if family == "train_channel":
        batch, kind = rng.choice([1, 2, 4]), rng.choice(["kda", "kda", "gdn2"])
        n = _length(rng, 64, _fit(16384, batch))
        return _case(None, "train", kind, batch, n, heads, 128, 128, docs=rng.choice(["none", "segments"]), lo=min(64, n),
                     hi=n, l2norm=rng.random() < 0.5)
    if family == "train_ssd":
        batch = rng.choice([1, 2, 4, 8])
        n = _length(rng, 64, _fit(16384, batch))
        return _case(None, "train", "ssd", batch, n, rng.choice([24, 32, 64]), 128, 64, Hk=rng.choice([1, 1, 8]), dtype=dtype,
                     docs=rng.choice(["none", "segments"]), lo=min(64, n), hi=n)
    if family == "layer":
        batch = rng.choice([1, 2, 4, 8])
        n = _length(rng, 64, _fit(16384, batch))
        return _case(None, "layer", "gated_deltanet", batch, n, rng.choice([4, 8, 16]), 128, rng.choice([128, 128, 256]),
                     dtype=dtype, docs=rng.choice(["none", "segments"]), lo=min(64, n), hi=n)
    if family == "f32":
        k = rng.choice([64, 64, 128])
        return _case(None, "train", rng.choice(["gated_deltanet", "gated_deltanet", "simple_gla", "kda"]), rng.choice([1, 2]),
                     _log_int(rng, 32, 512 if k == 128 else 1024), rng.choice([2, 4, 8]), k, k, dtype="f32",
                     docs=rng.choice(["none", "segments"]), lo=16, hi=256)
    n = _log_int(rng, 12288, 98304)
    return _case(None, "train", "gated_deltanet", 1, n, heads, 128, 128, docs=rng.choice(["none", "segments"]),
                 lo=min(4096, n), hi=n)


class _Source:
    """Seeded inputs on the GPU; lengths of documents come from a host generator of the same seed."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)
        self.host = random.Random(seed)

    def normal(self, *shape):
        return torch.randn(*shape, generator=self.gen, device="cuda", dtype=torch.float32)

    def uniform(self, lo, hi, *shape):
        return torch.rand(*shape, generator=self.gen, device="cuda", dtype=torch.float32) * (hi - lo) + lo

    def unit(self, *shape):
        x = self.normal(*shape)
        return x * torch.rsqrt((x * x).sum(-1, keepdim=True) + 1e-6)

    def documents(self, c):
        """``segment_ids [B, T]``: every row cut into documents of lo .. hi tokens (the last one takes what is left)."""
        rows = []
        for _ in range(c["B"]):
            lengths, left = [], c["T"]
            while left > 0:
                n = min(left, self.host.randint(c["lo"], c["hi"]))
                lengths.append(n)
                left -= n
            rows.append(torch.repeat_interleave(torch.arange(len(lengths)), torch.tensor(lengths)))
        return torch.stack(rows).to(device="cuda", dtype=torch.int32)

    def prompts(self, c):
        """``cu_seqlens [seqs + 1]``: ``seqs`` prompts of random lengths, none of them empty, that fill T tokens."""
        cuts = sorted(self.host.sample(range(1, c["T"]), c["seqs"] - 1))
        return torch.tensor([0, *cuts, c["T"]], device="cuda", dtype=torch.int32)


def _gates(src, c):
    """Gate inputs of the op: log-decays that keep most of the state per token, write strengths in (0, 1)."""
    shape = (c["B"], c["T"], c["H"])
    td = DTYPES[c["dtype"]]
    if c["kind"] in ("kda", "gdn2"):
        gates = {"g": torch.nn.functional.logsigmoid(src.normal(*shape, c["K"]) + 4.0) / 8.0}
    elif c["kind"] == "deltanet":
        gates = {}
    else:
        gates = {"g": torch.nn.functional.logsigmoid(src.normal(*shape) + 3.0)}
    if c["kind"] == "gdn2":
        gates["b"] = torch.sigmoid(src.normal(*shape, c["K"])).to(td)
        gates["w"] = torch.sigmoid(src.normal(*shape, c["V"])).to(td)
    elif c["kind"] != "simple_gla":
        gates["beta"] = torch.sigmoid(src.normal(*shape))
    return gates


def _mamba_gate_parameters(src, heads):
    dt = torch.exp(src.uniform(math.log(0.001), math.log(0.1), heads))
    return torch.log(src.uniform(1.0, 16.0, heads)), torch.log(torch.expm1(dt))  # A_log, dt_bias


def prepare(case, seed):
    c = case
    src = _Source(seed)
    td = DTYPES[c["dtype"]]
    B, T, H, Hk, K, V = (c[n] for n in ("B", "T", "H", "Hk", "K", "V"))
    x, options = {}, {}
    if c["docs"] == "segments":
        options["segment_ids"] = src.documents(c)
    elif c["docs"] == "rows":
        options["cu_seqlens"] = src.prompts(c)
    if c["mode"] == "layer":
        for n, width in (("q", H * K), ("k", H * K), ("v", H * V)):
            x[n] = src.normal(B, T, width).to(td)
            x["conv_" + n] = src.uniform(-0.5, 0.5, width, 4)
        x["a"], x["b"] = src.normal(B, T, H).to(td), src.normal(B, T, H).to(td)
        x["A_log"], x["dt_bias"] = _mamba_gate_parameters(src, H)
        x["z"] = src.normal(B, T, H, V).to(td)
        x["norm"] = torch.ones(V, device="cuda")
    elif c["kind"] == "ssd":
        a_log, dt_bias = _mamba_gate_parameters(src, H)
        x["x"] = src.normal(B, T, H, V).to(td)
        x["dt"] = torch.nn.functional.softplus(src.normal(B, T, H) + dt_bias)
        x["a"] = -torch.exp(a_log)
        x["b"] = (src.normal(B, T, Hk, K) / K ** 0.5).to(td)
        x["c"] = (src.normal(B, T, Hk, K) / K ** 0.5).to(td)
        x["d"] = src.normal(H)
    else:
        direction = src.normal if c["l2norm"] else src.unit  # the op normalises q and k itself, or they come normalised
        x["q"], x["k"] = direction(B, T, Hk, K).to(td), direction(B, T, Hk, K).to(td)
        x["v"] = src.normal(B, T, H, V).to(td)
        x.update(_gates(src, c))
        if c["l2norm"]:
            options["use_qk_l2norm"] = True
    if c["state"]:
        rows = c["seqs"] if c["docs"] == "rows" else B
        x["initial_state"] = src.normal(rows, H, K, V) / K ** 0.5
    state = {"case": c, "x": x, "options": options}
    if c["mode"] in ("train", "layer"):
        for t in x.values():
            t.requires_grad_(True)
        state["d_o"] = src.normal(B, T, H, V).to(td)
    else:
        options["output_final_state"] = True
    return state


def _layer(x, options, heads, head_dim):
    seg = options.get("segment_ids")
    q, _ = short_conv(x["q"], x["conv_q"], head_dim=head_dim, segment_ids=seg)
    k, _ = short_conv(x["k"], x["conv_k"], head_dim=head_dim, segment_ids=seg)
    v, _ = short_conv(x["v"], x["conv_v"], segment_ids=seg)
    g, beta = gate_prologue(x["a"], x["A_log"], x["dt_bias"], x["b"])
    shape = (*q.shape[:2], heads, -1)
    o, _ = ops.linear_attention("gated_deltanet", q.view(shape), k.view(shape), v.view(shape), g=g, beta=beta, **options)
    return gated_rms_norm(o, x["z"], x["norm"])


def run(state):
    c, x, options = state["case"], state["x"], state["options"]
    if c["mode"] == "layer":
        o, final = _layer(x, options, c["H"], c["K"]), None
    elif c["kind"] == "ssd":
        o, final = mamba2_ssd(**x, **options)
    else:
        o, final = ops.linear_attention(c["kind"], **x, **options)
    if c["mode"] in ("step", "prefill"):
        return {"o": o, "final_state": final}
    grads = torch.autograd.grad(o, list(x.values()), state["d_o"])
    return {"o": o.detach(), **{"d_" + n: t for n, t in zip(x, grads)}}


def _elements(c):
    """Bytes of every input and output tensor of one forward, and of the state rows."""
    B, T, H, Hk, K, V = (c[n] for n in ("B", "T", "H", "Hk", "K", "V"))
    es = DTYPES[c["dtype"]].itemsize
    tok = B * T
    inputs = 2 * tok * Hk * K * es + tok * H * V * es
    if c["mode"] == "layer":
        inputs += 2 * tok * H * es + tok * H * V * es  # a, b and z; the parameters are negligible
    elif c["kind"] in ("kda", "gdn2"):
        inputs += tok * H * K * 4 + (tok * H * (K + V) * es if c["kind"] == "gdn2" else tok * H * 4)
    elif c["kind"] in ("gated_deltanet",):
        inputs += 2 * tok * H * 4
    else:
        inputs += tok * H * 4
    state = (c["seqs"] if c["docs"] == "rows" else B) * H * K * V * 4
    return inputs, tok * H * V * es, state


def work(case):
    """Every input read once and every output written once; the products of the chunked algorithm (chunks of 64 tokens)
    forward, and twice as many backward. The inverse of a chunk's triangular matrix is not counted."""
    c = case
    inputs, output, state = _elements(c)
    rows = 4 * c["B"] * c["T"] if c["docs"] == "segments" else 0
    nbytes = inputs + output + rows
    if c["mode"] in ("train", "layer"):
        nbytes += inputs + output  # the upstream gradient, and a gradient of every input
        nbytes += 2 * state if c["state"] else 0
    else:
        nbytes += state * (2 if c["state"] else 1)
    chunk = min(64, c["T"])
    delta = c["kind"] not in ("simple_gla", "ssd")
    K, V = c["K"], c["V"]
    per_token = chunk * K * c["Hk"] / c["H"] + chunk * V + 2 * K * V  # scores, their product with v, read, update
    if delta:
        per_token += chunk * K * c["Hk"] / c["H"] + chunk * V + K * V  # k k^T, the solve's product, recall
    flops = 2 * per_token * c["B"] * c["T"] * c["H"] * (3 if c["mode"] in ("train", "layer") else 1)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Measured against the float32 token scan on the same inputs (float32: against the chunked algorithm in 64 bits), over
    the listed cases and 28 drawn ones: bf16 up to 0.004 with scalar gates, 0.006 with gates per channel, 0.008 for the
    gate parameters of a layer; f16 up to 0.0008; float32 up to 1e-6."""
    return {"rel": {"bf16": 1.5e-2, "f16": 3e-3, "f32": 1e-5}[case["dtype"]]}
