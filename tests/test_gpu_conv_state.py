"""The state a short convolution hands on, as one kernel where documents mask it: against the plain tensor form, bit for
bit (it is a masked copy), for sequences shorter and longer than the window."""

import pytest
import torch

from jax_linear_attention_b200.layers import short_conv
from jax_linear_attention_b200.layers.conv import _final_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("T,K", [(1, 4), (2, 4), (3, 4), (4, 4), (65, 4), (2, 2), (5, 3)])
@pytest.mark.parametrize("with_state", [False, True])
def test_new_state_is_the_masked_tail(dtype, T, K, with_state):
    gen = torch.Generator("cuda").manual_seed(T * 7 + K)
    B, C = 3, 24
    x = torch.randn(B, T, C, generator=gen, device="cuda").to(dtype)
    w = torch.randn(C, K, generator=gen, device="cuda")
    state = torch.randn(B, K - 1, C, generator=gen, device="cuda").to(dtype) if with_state else None
    seg = torch.randint(0, 2, (B, T), generator=gen, device="cuda").cumsum(1)
    _, got = short_conv(x, w, segment_ids=seg, state=state)
    assert torch.equal(got, _final_state(x, state, seg, K))
