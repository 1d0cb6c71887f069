"""Decoding steps (one token per row, no gradient): the single-pass kernel against the float64 oracle, over head sizes,
kinds, key groups and dtypes, with and without a state on either side. The arithmetic is fp32, so 16-bit results differ
from the oracle's by the rounding of the outputs alone (bf16 2^-9 relative, f16 2^-12) and the state by fp32 rounding."""

import pytest
import torch

from oracle.cases import make_case
from tests._util import TORCH_DTYPE, compare, run_cuda, run_oracle

pytestmark = pytest.mark.gpu
TOL = {"bfloat16": 2.0 ** -9, "float16": 2.0 ** -12, "float32": 2e-6}


@pytest.mark.parametrize("kind", ["simple_gla", "deltanet", "gated_deltanet", "kda", "gdn2"])
@pytest.mark.parametrize("K,V", [(64, 64), (128, 128), (64, 128), (128, 64), (128, 256), (128, 512), (256, 128)])
def test_step_matches_oracle(kind, K, V):
    if kind == "gdn2" and V > 256:
        pytest.skip("calls with a read key keep V <= 256")
    dtype = {64: "float16", 128: "bfloat16", 256: "float32"}[K]
    case = make_case(kind, B=3, T=1, H=4, Hk=4 if kind == "gdn2" else 2, K=K, V=V, seed=K + V, dtype=dtype, h0=True)
    want = run_oracle(kind, case, scale=case["meta"]["scale"], grads=False)
    got = run_cuda(kind, case, scale=case["meta"]["scale"], dtype=dtype, grads=False)
    compare({"o": got["o"]}, {"o": want["o"]}, TOL[dtype], f"{kind} o")
    # gdn2's operands k * b and v * w are rounded to the tensors' dtype before the kernel
    compare({"ht": got["ht"]}, {"ht": want["ht"]}, TOL[dtype] if kind == "gdn2" else 2e-6, f"{kind} state")


def test_step_norm_and_unaligned_state():
    from jax_linear_attention_b200 import ops

    case = make_case("gated_deltanet", B=2, T=1, H=2, K=128, V=128, seed=5, dtype="bfloat16", h0=True)
    want = run_oracle("gated_deltanet", case, scale=case["meta"]["scale"], grads=False, l2norm=True)
    t = {n: torch.tensor(case[n], device="cuda") for n in ("q", "k", "v", "g", "beta", "h0")}
    pad = torch.zeros(t["h0"].numel() + 1, device="cuda")
    pad[1:] = t["h0"].flatten()
    q, k, v = (t[n].to(torch.bfloat16) for n in ("q", "k", "v"))
    o, ht = ops.linear_attention("gated_deltanet", q, k, v, g=t["g"], beta=t["beta"], scale=case["meta"]["scale"],
                                 initial_state=pad[1:].view_as(t["h0"]), output_final_state=True, use_qk_l2norm=True)
    # the normalised q and k are rounded to bf16 (as the reference rounds them)
    compare({"o": o.float().cpu().numpy(), "ht": ht.cpu().numpy()}, want, 2.0 ** -8, "norm")


@pytest.mark.parametrize("dtype,groups,skip", [("bfloat16", 1, True), ("float16", 4, False)])
def test_ssd_step_matches_general_form(dtype, groups, skip):
    """The fused step against the same call with gradients on, which takes the glue and chunk kernels."""
    from jax_linear_attention_b200.layers import mamba2_ssd

    gen = torch.Generator("cuda").manual_seed(3)
    td = TORCH_DTYPE[dtype]
    B, H, P, N = 3, 8, 64, 128
    def normal(*s):
        return torch.randn(*s, generator=gen, device="cuda")
    x, b, c = normal(B, 1, H, P).to(td), normal(B, 1, groups, N).to(td), (normal(B, 1, groups, N) / N ** 0.5).to(td)
    dt, a, h0 = torch.rand(B, 1, H, generator=gen, device="cuda") * 0.1, -1 - normal(H).abs(), normal(B, H, N, P)
    d = normal(H) if skip else None
    y, s = mamba2_ssd(x, dt, a, b, c, d=d, initial_state=h0, output_final_state=True)
    y2, s2 = mamba2_ssd(x.requires_grad_(True), dt, a, b, c, d=d, initial_state=h0, output_final_state=True)
    # the general form multiplies with a 16-bit copy of the state: its error is that rounding
    compare({"y": y.float().cpu().numpy(), "s": s.cpu().numpy()},
            {"y": y2.detach().float().cpu().numpy(), "s": s2.detach().cpu().numpy()},
            {"bfloat16": 2.0 ** -8, "float16": 2.0 ** -11}[dtype], "ssd step")


def test_step_of_more_rows_than_a_grid_dimension_holds():
    """65537 rows (gridDim.y ends at 65535): every row is its own step, so the last ones equal a call of their own."""
    from jax_linear_attention_b200 import ops

    gen = torch.Generator("cuda").manual_seed(9)
    B, K, V = 65537, 64, 64
    q, k, v = (torch.randn(B, 1, 1, 64, generator=gen, device="cuda").to(torch.bfloat16) for _ in range(3))
    g = -torch.rand(B, 1, 1, generator=gen, device="cuda")
    h0 = torch.randn(B, 1, K, V, generator=gen, device="cuda")
    o, ht = ops.linear_attention("simple_gla", q, k, v, g=g, initial_state=h0, output_final_state=True)
    tail = slice(B - 3, B)
    o3, ht3 = ops.linear_attention("simple_gla", q[tail], k[tail], v[tail], g=g[tail], initial_state=h0[tail],
                                   output_final_state=True)
    assert torch.equal(o[tail], o3) and torch.equal(ht[tail], ht3)
    want = torch.exp(g)[..., None] * h0 + k.float().transpose(-1, -2) * v.float()
    assert torch.allclose(ht, want, rtol=1e-5, atol=1e-6)  # (one exp, one product and one sum in fp32)
