"""CPU tests of the host's routing rules: what it asks of the library is looked at, nothing is launched."""

import pytest
import torch

from jax_linear_attention_b200 import _lib
from jax_linear_attention_b200.ops import cuda


@pytest.fixture
def launches(monkeypatch):
    """The calls that would have been launched: ``(entry point, arguments)``."""
    calls = []
    monkeypatch.setattr(_lib, "launch", lambda name, device, *args: calls.append((name, args)))
    return calls


def _prologues(launches):
    """Per forward: whether it relies on an earlier prologue, and the buffer that holds the tables."""
    forwards = [args for name, args in launches if name == "jla_linear_attention_fwd"]
    return [(bool(p.flags & _lib.FLAG_PREP_DONE), io.residuals or io.scratch) for p, io in forwards]


@pytest.mark.parametrize("kind,H,Hk", [("simple_gla", 8, 1), ("gated_deltanet", 2, 2)])
def test_shared_prologue_belongs_to_a_value_width(launches, kind, H, Hk):
    """The value width decides which kernels run and which tables the prologue leaves behind (values of 64 next to keys of
    128 and the 128 x 128 map pass of a split sequence share neither): a pass reuses the tables of its own width only, and
    finds them again after a pass of another width."""
    T, K = 128, 128
    q, k = torch.zeros(1, T, Hk, K, dtype=torch.bfloat16), torch.zeros(1, T, Hk, K, dtype=torch.bfloat16)
    g, beta = torch.zeros(1, T, H), None if kind == "simple_gla" else torch.zeros(1, T, H)
    cfg = dict(kind=kind, scale=1.0, l2norm=False, precision=None, output_final_state=True, cu_seqlens=None,
               segment_ids=None, prep_owners=(k, g, beta, None, None, None))
    narrow, wide = (torch.zeros(1, T, H, V, dtype=torch.bfloat16) for V in (64, 128))
    with cuda.shared_prep():
        for v, needs_grad in ((narrow, False), (wide, False), (narrow, True), (wide, False)):
            cuda._forward(q, k, v, g, beta, None, None, cfg, needs_grad)
    (done0, narrow0), (done1, wide1), (done2, narrow2), (done3, wide3) = _prologues(launches)
    assert [done0, done1, done2, done3] == [False, False, True, True]
    assert narrow2 == narrow0 and wide3 == wide1 and narrow0 != wide1


@pytest.mark.parametrize("kind,V,l2norm", [("kda", 128, False), ("simple_gla", 64, False), ("gated_deltanet", 128, True)])
def test_shared_prologue_belongs_to_its_queries(launches, monkeypatch, kind, V, l2norm):
    """Where the prologue works on q too (KDA folds the gates into it, simple GLA's score table, the in-op norm), another q
    means another prologue."""
    T, H, K = 128, 4, 128
    monkeypatch.setattr(torch.Tensor, "is_cuda", property(lambda self: True), raising=False)
    q, q2, k = (torch.zeros(1, T, 2 if kind == "simple_gla" else H, K, dtype=torch.bfloat16) for _ in range(3))
    v = torch.zeros(1, T, H, V, dtype=torch.bfloat16)
    g = torch.zeros(1, T, H, K) if kind == "kda" else torch.zeros(1, T, H)
    beta = None if kind == "simple_gla" else torch.zeros(1, T, H)
    with cuda.shared_prep():
        for x in (q, q, q2):
            cuda._run(kind, x, k, v, g, beta, scale=1.0, initial_state=None, output_final_state=True, cu_seqlens=None,
                      segment_ids=None, use_qk_l2norm=l2norm)
    assert [done for done, _ in _prologues(launches)] == [False, True, False]


def _step_inputs(B, H, Hk, K, V):
    q, k = torch.empty(B, 1, Hk, K, dtype=torch.bfloat16), torch.empty(B, 1, Hk, K, dtype=torch.bfloat16)
    return q, k, torch.empty(B, 1, H, V, dtype=torch.bfloat16), torch.empty(B, 1, H)


@pytest.mark.parametrize("B", [0, 1, 65535, 65536])
def test_decoding_steps_of_any_batch(launches, monkeypatch, B):
    """A batch of any size runs: as one pass over the state from one row on, as the general call without rows."""
    from jax_linear_attention_b200 import ops
    from jax_linear_attention_b200.layers import mamba2_ssd

    monkeypatch.setattr(torch.Tensor, "is_cuda", property(lambda self: True), raising=False)
    lib = _lib.load()
    for V in (256, 384, 512):  # wide value heads: the step kernel takes them whole
        q, k, v, g = _step_inputs(B, 1, 1, 64, V)
        ops.linear_attention("simple_gla", q, k, v, g=g)
        p = launches[-1][1][0]
        assert (p.B, p.H * p.V, p.V) == (B, V, V if B else 128)
        assert lib.jla_fwd_scratch_bytes(p) == 0 if B else True
        p.q = p.k = p.v = p.g = None
        assert lib.jla_linear_attention_fwd(p, _lib.FwdIO(), None) == (_lib.ERR_BAD_ARGUMENT if B else _lib.OK)  # (no pointers)
    launches.clear()
    c, b, x, dt = _step_inputs(B, 1, 1, 64, 64)
    mamba2_ssd(x, dt, torch.empty(1), b, c)
    assert [name for name, _ in launches] == (["jla_ssd_step"] if B else ["jla_ssd_inputs_fwd", "jla_linear_attention_fwd"])
    if B:
        p = launches[0][1][0]
        assert lib.jla_unsupported_reason(p) is None and lib.jla_fwd_scratch_bytes(p) == 0


def test_one_token_of_mamba2_is_a_step_only_where_nobody_could_tell(launches, monkeypatch):
    """The fused step goes past autograd and past the table of implementations, so it leaves forward-mode tangents,
    transforms, tensor subclasses and a replaced implementation to the general form; no_grad calls of parameters are steps."""
    import torch.autograd.forward_ad as fwd

    from jax_linear_attention_b200 import ops
    from jax_linear_attention_b200.layers import mamba2_ssd

    monkeypatch.setattr(torch.Tensor, "is_cuda", property(lambda self: True), raising=False)
    c, b, x, dt = _step_inputs(2, 1, 1, 64, 64)
    a = torch.nn.Parameter(-torch.ones(1))

    def names(*args):
        launches.clear()
        mamba2_ssd(*args)
        return [name for name, _ in launches]

    general = ["jla_ssd_inputs_fwd", "jla_linear_attention_fwd"]
    with torch.no_grad():
        assert names(x, dt, a, b, c) == ["jla_ssd_step"]
        assert names(x, dt, a, b.as_subclass(type("Labelled", (torch.Tensor,), {})), c) == general
    assert names(x, dt, a, b, c) == general  # a requires a gradient
    with fwd.dual_level():
        with pytest.raises(NotImplementedError):  # as the general form has always answered
            names(fwd.make_dual(x, torch.ones_like(x)), dt, a.detach(), b, c)
        assert not any(name == "jla_ssd_step" for name, _ in launches)
    with pytest.raises(RuntimeError):  # (the general form's autograd function has no rule for vmap)
        torch.vmap(lambda x: mamba2_ssd(x, dt, a.detach(), b, c)[0])(x[None])
    entry = ops._REGISTRY["cuda"]["simple_gla"]
    calls = []
    ops.register("cuda", "simple_gla", lambda *args, **kw: calls.append(kw) or entry[0](*args, **kw), entry[1], auto=True)
    try:
        assert names(x, dt, a.detach(), b, c) == general and len(calls) == 1
    finally:
        ops._REGISTRY["cuda"]["simple_gla"] = entry
    assert names(x, dt, a.detach(), b, c) == ["jla_ssd_step"]


def test_a_split_call_runs_in_inference_mode(launches, monkeypatch):
    """The three passes of a split sequence on inference tensors: no graph, and every pass makes its own tables (such tensors
    have no version that an update in place would change)."""
    from jax_linear_attention_b200.distributed import context_parallel as cp

    monkeypatch.setattr(torch.Tensor, "is_cuda", property(lambda self: True), raising=False)
    monkeypatch.setattr(cp, "piece_scan", lambda *args, **kw: None)
    with torch.inference_mode():
        q, k, v = (torch.zeros(1, 1000, 2, 128, dtype=torch.bfloat16) for _ in range(3))
        g, beta = torch.zeros(1, 1000, 2), torch.zeros(1, 1000, 2)
    for mode in (torch.inference_mode, torch.no_grad):  # (inference tensors leave the mode as what they are)
        launches.clear()
        with mode():
            o, ht = cp.context_parallel_linear_attention("gated_deltanet", q, k, v, g=g, beta=beta, group=False, piece_len=256,
                                                         impl="cuda", output_final_state=True)
        assert o.shape == v.shape and ht.shape == (1, 2, 128, 128) and not o.requires_grad
        assert [done for done, _ in _prologues(launches)] == [False] * 3
