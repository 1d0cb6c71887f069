"""The token scan at the edges of its staging (8 tokens), checkpoint blocks (16 tokens), channel tiles (64) and key-lane
layouts (K <= 32, 64, 128, 256), forward and gradients against the float64 oracle. fp32 arithmetic: the relative error
per tensor stays around 2e-7 (2^-24 per operation, sums of a few hundred terms), far inside the 1e-5 of the fp32 bar;
2e-6 leaves a factor of ten for the decays' exponentials."""

import numpy as np
import pytest
import torch

from oracle.cases import make_case
from tests._util import compare, run_cuda, run_oracle

pytestmark = pytest.mark.gpu
TOL = 2e-6


@pytest.mark.parametrize("kind", ["simple_gla", "deltanet", "gated_deltanet", "kda", "gdn2"])
@pytest.mark.parametrize("T,K,V", [(1, 64, 64), (7, 8, 32), (8, 32, 8), (9, 40, 64), (15, 24, 64), (16, 64, 16), (17, 72, 32),
                                   (31, 128, 256), (33, 256, 128), (65, 128, 8), (40, 256, 256)])
def test_scan_edges(kind, T, K, V):
    case = make_case(kind, B=2, T=T, H=2, Hk=2 if kind == "gdn2" else 1, K=K, V=V, seed=T + K + V, dtype="float32",
                     docs="mixed" if T > 8 else None, h0=True)
    want = run_oracle(kind, case, scale=case["meta"]["scale"])
    got = run_cuda(kind, case, scale=case["meta"]["scale"], dtype="float32")
    compare(got, want, TOL, f"{kind} {T} {K} {V}")


def test_rows_of_every_length_share_the_checkpoints():
    """Packed rows of 0, 1, 8, 15, 16, 17, 48 and 3 tokens: every row has its own checkpoints and states."""
    cu = np.cumsum([0, 0, 1, 8, 15, 16, 17, 48, 0, 3])
    case = make_case("kda", B=1, T=int(cu[-1]), H=3, K=64, V=64, seed=3, dtype="float32")
    rng = np.random.default_rng(7)
    case["h0"] = rng.standard_normal((len(cu) - 1, 3, 64, 64)).astype(np.float32)
    case["dht"] = rng.standard_normal((len(cu) - 1, 3, 64, 64)).astype(np.float32)
    want = run_oracle("kda", case, scale=0.125, cu_seqlens=cu)
    got = run_cuda("kda", case, scale=0.125, dtype="float32", cu_seqlens=cu.astype(np.int32))
    compare(got, want, TOL, "rows")


@pytest.mark.parametrize("kind", ["simple_gla", "gated_deltanet", "kda", "gdn2"])
def test_gate_gradients_entry_by_entry_behind_strong_decays(kind):
    """Decays of e^-12 and e^-0.05 in turn: dg of a strongly decaying token is a sum of terms that all carry its decay, so
    its entries are as exact as fp32 sums (2^-24 per operation, cancellation among a few thousand terms: a median around
    2e-7; the largest tensor entries say nothing about them). Without an entering state dg of a row's first token is zero."""
    case = make_case(kind, B=2, T=64, H=2, K=64, V=64, seed=17, dtype="float32")
    rng = np.random.default_rng(17)
    strong = (np.arange(64) % 2 == 0).reshape(1, 64, *[1] * (case["g"].ndim - 2))
    case["g"] = (np.where(strong, -12.0, -0.05) * rng.uniform(0.9, 1.1, case["g"].shape)).astype(np.float32)
    want = run_oracle(kind, case, scale=case["meta"]["scale"])
    got = run_cuda(kind, case, scale=case["meta"]["scale"], dtype="float32")
    compare(got, want, TOL, kind)
    assert (got["dg"][:, 0] == 0).all()
    err = np.abs(got["dg"][:, 1:] - want["dg"][:, 1:]) / np.abs(want["dg"][:, 1:])
    assert np.median(err) < 2e-6, np.median(err)


def test_heads_in_slices_are_the_heads_of_calls_of_their_own():
    """Checkpoints of more than 32 GiB: 33 heads of 256 x 256 over 1024 rows run as slices of 17 and 16 heads through the same
    buffers, with the results of two calls of 17 and 16 heads, bit for bit."""
    from jax_linear_attention_b200 import ops

    gen = torch.Generator("cuda").manual_seed(4)
    B, T, H, K = 1024, 16, 33, 256

    def normal(*shape):
        return torch.randn(*shape, generator=gen, device="cuda") / 16

    x = [normal(B, T, H, K) for _ in range(3)] + [-normal(B, T, H).abs(), torch.sigmoid(normal(B, T, H))]
    do = normal(B, T, H, K)

    def gradients(heads):
        leaves = [t[:, :, heads].contiguous().requires_grad_(True) for t in x]
        o, _ = ops.linear_attention("gated_deltanet", *leaves[:3], g=leaves[3], beta=leaves[4], scale=1.0)
        return torch.autograd.grad(o, leaves, do[:, :, heads])

    parts = [torch.cat(p, 2) for p in zip(gradients(slice(0, 17)), gradients(slice(17, 33)))]
    for whole, part in zip(gradients(slice(0, 33)), parts):
        assert torch.equal(whole, part)
