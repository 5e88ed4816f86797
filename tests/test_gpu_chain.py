"""The one-launch chain of steps from a floating-point state against the same tokens as separate steps from
``init_quant_state`` (eager torch): equal bit for bit, at the edges of a chunk of tokens (8) and of a launch (1024)."""

from __future__ import annotations

import pytest
import torch

from carrykernel_b200.statequant import kernel as sq

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("B,HV,T", [(1, 1, 1), (2, 3, 7), (1, 2, 8), (3, 32, 9), (1, 1, 1025)])
@pytest.mark.parametrize("res_fmt", [sq.RES_FP32, sq.RES_FP16, sq.RES_FP8])
@pytest.mark.parametrize("dtype,bits", [(torch.float32, 8), (torch.bfloat16, 3)])
def test_chain_equals_separate_steps(B, HV, T, res_fmt, dtype, bits):
    from carrykernel_b200 import _lib
    K = V = 128
    g = torch.Generator().manual_seed(T)
    h0 = (torch.randn(B, HV, K, V, generator=g) * 0.1).to(DEV)
    h0[0, 0, :, 3] = 0.0                              # a column at the scale floor
    q, k = (torch.nn.functional.normalize(torch.randn(T, B, HV, K, generator=g), dim=-1).to(DEV, dtype) for _ in range(2))
    v = torch.randn(T, B, HV, V, generator=g).to(DEV, dtype)
    alpha, beta = (torch.rand(T, B, HV, generator=g).to(DEV) * 0.2 + x for x in (0.8, 0.3))
    o, codes, scale, e, e_scale = sq.gdn_quant_decode_fused(h0, q, k, v, alpha, beta, T, bits=bits, res_fmt=res_fmt)
    assert _lib.load_library().carry_gdn_last_kernel() == 7 and e_scale is None
    state = sq.init_quant_state(h0, bits, res_fmt)
    for t in range(T):
        ot, *state = sq.gdn_quant_step_fused(*state, q[t], k[t], v[t], alpha[t], beta[t], bits=bits, res_fmt=res_fmt)
        assert torch.equal(o[t], ot), f"token {t}"
    for got, want in zip((codes, scale, e), state):
        assert torch.equal(got.float(), want.float())


@pytest.mark.parametrize("res_fmt", [sq.RES_FP32, sq.RES_FP16, sq.RES_FP8])
def test_chain_keeps_what_is_not_a_number(res_fmt):
    """A column of h0 with a NaN or an infinity: its scale, and with it the first output, is what torch makes of it."""
    K = V = 128
    g = torch.Generator().manual_seed(7)
    h0 = (torch.randn(1, 2, K, V, generator=g) * 0.1).to(DEV)
    h0[0, 0, 100, 5], h0[0, 0, 0, 9], h0[0, 1, 127, 0] = float("nan"), float("inf"), float("-inf")
    q, k = (torch.nn.functional.normalize(torch.randn(2, 1, 2, K, generator=g), dim=-1).to(DEV) for _ in range(2))
    v = torch.randn(2, 1, 2, V, generator=g).to(DEV)
    alpha, beta = (torch.rand(2, 1, 2, generator=g).to(DEV) * 0.2 + x for x in (0.8, 0.3))
    plain = lambda x: x.float().nan_to_num(nan=12345.0)  # noqa: E731
    o, *got = sq.gdn_quant_decode_fused(h0, q, k, v, alpha, beta, 2, res_fmt=res_fmt)
    state = sq.init_quant_state(h0, 8, res_fmt)
    for t in range(2):
        ot, *state = sq.gdn_quant_step_fused(*state, q[t], k[t], v[t], alpha[t], beta[t], res_fmt=res_fmt)
        assert torch.equal(plain(o[t]), plain(ot)), f"token {t}"
    assert bool(o[0, 0, 0, [5, 9]].isnan().all()) and bool(o[0, 0, 1, 0].isnan())
    for x, y in zip(got[:3], state[:3]):
        assert torch.equal(plain(x), plain(y))
