"""The split training kernels (head sizes other than K = V = 128) on both sides of their size rules: value blocks of 32 and
64 columns (few and many chains), walks of one and of eight heads, ragged last chunks, documents inside chunks, initial
and final states. Reference: the fp32 token scan on the same 16-bit tensors, itself held to the float64 oracle. The error
is that of 16-bit operands and outputs (bf16: 2^-9 per rounding, a few roundings in a row; f16 an eighth of that)."""

import pytest
import torch

from oracle.cases import make_case
from jax_linear_attention_b200 import _lib
from tests._util import cabi_fwd_bwd, compare, run_cuda, run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,B,T,H,Hk,K,V,dtype", [
    ("simple_gla", 10, 130, 64, 1, 128, 64, "bfloat16"),   # 640 chains, walks of eight heads
    ("simple_gla", 1, 65, 8, 1, 128, 64, "float16"),       # few chains, one head a CTA
    ("simple_gla", 2, 63, 4, 2, 64, 128, "bfloat16"),
    ("gated_deltanet", 20, 129, 32, 16, 64, 64, "bfloat16"),  # 640 chains
    ("gated_deltanet", 2, 1, 2, 1, 64, 64, "float16"),
    ("deltanet", 3, 191, 4, 4, 128, 64, "float16"),
    ("gated_deltanet", 10, 70, 32, 32, 64, 128, "bfloat16"),
    ("gated_deltanet", 1, 64, 40, 5, 128, 64, "bfloat16"),
])
def test_split_passes_match_the_scan(kind, B, T, H, Hk, K, V, dtype):
    case = make_case(kind, B=B, T=T, H=H, Hk=Hk, K=K, V=V, seed=B + T, dtype=dtype, docs="mixed" if T > 8 else None, h0=True)
    want = run_cuda(kind, case, scale=case["meta"]["scale"], dtype=dtype, precision="highest")
    got = run_cuda(kind, case, scale=case["meta"]["scale"], dtype=dtype)
    compare(got, want, {"bfloat16": 1e-2, "float16": 2e-3}[dtype], f"{kind} B{B} T{T} H{H} K{K} V{V}")


@pytest.mark.parametrize("kind,dO", [("gated_deltanet", 1.0), ("gated_deltanet", 1e-3), ("simple_gla", 1.0)])
def test_float16_state_gradient_behind_a_strong_decay(kind, dO):
    """A chunk that starts behind e^-8: what its queries send back to the entering state is that factor times a sum of 64
    products, every factor of them a normal f16 number (unit rows / 8, upstream gradients of 1 and of 1e-3). So dh0 is off
    by the rounding of the weighted operand (2^-11 an element, averaged over the sum); without writes (beta = 0) nothing
    else reaches it."""
    import numpy as np

    case = make_case(kind, B=2, T=64, H=2, K=64, V=64, seed=5, dtype="float16", h0=True)
    case["q"] = case["q"] / 4  # rows of length 4 otherwise
    case["g"] = np.full_like(case["g"], -0.01)
    case["g"][:, 0] = -8.0
    if "beta" in case:
        case["beta"] = np.zeros_like(case["beta"])
    case["dht"] = np.zeros_like(case["dht"])
    case["do"] = (case["do"] * dO).astype(np.float16).astype(np.float32)
    want = run_oracle(kind, case, scale=case["meta"]["scale"])
    got = run_cuda(kind, case, scale=case["meta"]["scale"], dtype="float16")
    compare({"dh0": got["dh0"]}, {"dh0": want["dh0"]}, 2.0 ** -11, f"{kind} {dO}")


@pytest.mark.parametrize("H,Hk,K", [(8, 1, 128), (8, 2, 64)])
def test_float16_head_sums_beyond_the_range_of_one_head(H, Hk, K):
    """Upstream gradients of one sign over a group of heads: each head's dP stays inside f16 (64 * 1 * 300 = 19200), their sum
    does not. dq and dk, which are small because the keys and queries are, come out as of the fp32 scan. (So small queries and
    keys make o and the in-chunk part of dv subnormal f16 numbers: those two are only held to be finite.)"""
    import numpy as np

    case = make_case("simple_gla", B=1, T=130, H=H, Hk=Hk, K=K, V=64, seed=6, dtype="float16", h0=True)
    case["q"], case["k"] = case["q"] / 256, case["k"] / 256
    case["v"], case["do"] = np.ones_like(case["v"]), np.full_like(case["do"], 300.0)
    case["g"] = np.full_like(case["g"], -0.01)
    case["h0"], case["dht"] = case["h0"] / 256, case["dht"] / 256
    want = run_cuda("simple_gla", case, scale=1.0, dtype="float16", precision="highest")
    got = run_cuda("simple_gla", case, scale=1.0, dtype="float16")
    assert all(np.isfinite(x).all() for x in got.values())
    compare(got, {n: x for n, x in want.items() if n not in ("o", "dv")}, 2e-3, f"{H} {Hk} {K}")


@pytest.mark.parametrize("H,Hk,K,dtype", [(16, 2, 64, "bfloat16"), (8, 2, 64, "float16"), (6, 3, 64, "bfloat16"),
                                          (4, 2, 128, "float16"), (3, 1, 64, "bfloat16")])
def test_walks_over_eight_four_two_and_one_heads_of_a_group(H, Hk, K, dtype):
    """The gradients without the delta rule, for every length of a walk over the heads of a key group and both key sizes."""
    case = make_case("simple_gla", B=2, T=130, H=H, Hk=Hk, K=K, V=64, seed=H + K, dtype=dtype, docs="mixed", h0=True)
    want = run_cuda("simple_gla", case, scale=case["meta"]["scale"], dtype=dtype, precision="highest")
    got = run_cuda("simple_gla", case, scale=case["meta"]["scale"], dtype=dtype)
    compare(got, want, {"bfloat16": 1e-2, "float16": 2e-3}[dtype], f"{H} {Hk} {K}")


@pytest.mark.parametrize("kind", ["simple_gla", "kda"])
def test_outputs_that_are_not_16_byte_aligned(kind):
    """Where the kernels store 16 bytes out of their accumulators, a buffer at an odd multiple of four bytes takes the narrow
    stores: the same values (dv of the split kernels, dq and dk of KDA's)."""
    K, V = (128, 64) if kind == "simple_gla" else (128, 128)
    case = make_case(kind, B=2, T=100, H=2, K=K, V=V, seed=12, dtype="bfloat16", docs="mixed",
                     gates="kda_baseline" if kind == "kda" else "baseline")
    out = cabi_fwd_bwd(kind, case, scale=case["meta"]["scale"])
    t, p, dev = out["tensors"], out["problem"], out["o"].device

    def buffer(like, shift):  # `shift` elements behind a 16-byte boundary
        return torch.empty(like.numel() + 8, dtype=like.dtype, device=dev)[shift:][:like.numel()].view(like.shape)

    got = {n: buffer(out[n], 2 if n in (("dv",) if kind == "simple_gla" else ("dq", "dk")) else 0)
           for n in ("dq", "dk", "dv", "dg", "dbeta", "dh0") if out[n] is not None}
    assert any(x.data_ptr() % 16 == 4 for x in got.values())
    scratch = torch.empty_like(out["bwd_scratch"])
    io = _lib.BwdIO(t["do"].data_ptr(), t["dht"].data_ptr() if "dht" in t else None,
                    *(got[n].data_ptr() if n in got else None for n in ("dq", "dk", "dv", "dg", "dbeta", "dh0")),
                    out["residuals"].data_ptr(), out["residuals"].numel(), scratch.data_ptr(), scratch.numel())
    _lib.launch("jla_linear_attention_bwd", dev, p, io)
    for name, x in got.items():
        assert torch.equal(x, out[name]), name
