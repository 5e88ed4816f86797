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
