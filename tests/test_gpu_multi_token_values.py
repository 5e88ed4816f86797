"""Multi-token call against single-token calls, bit for bit, on activations that are zero, far apart in size, not finite or the
same for 96 tokens (the state under an int8 residual settles at rounding ties then, which have to be decided again): the two kernels
split a tile differently, and must still take every sum and maximum alike."""

from __future__ import annotations

import pytest
import torch

from oracle import gdn_oracle as orc
from parity import make_packed_inputs

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _same(x, y):
    x, y = x.float(), y.float()
    return torch.equal(torch.isnan(x), torch.isnan(y)) and torch.equal(torch.nan_to_num(x, 7.0), torch.nan_to_num(y, 7.0))


def _toks(T, B, H, HV, K, same, gain=1.0):
    return [list(make_packed_inputs(B, H, HV, K, K, seed=7 if same else 7 + t, qk_gain=gain)) for t in range(T)]


def _guarded(B, T, HV, K, dtype):
    """An output block with 32 elements on either side that nothing may write."""
    whole = torch.full((32 + B * T * HV * K + 32,), -3.0, dtype=dtype, device=DEV)
    return whole, whole[32:-32].view(B, T, HV, K)


def _check(toks, H, HV, K, resid_fmt, rscale, dtype, out_dtype, l2norm, rounds=1):
    from carrykernel_b200 import _lib
    from carrykernel_b200.vllm_integration import quantized_packed_decode as qpd
    B, T = toks[0][0].shape[0], len(toks)
    g = torch.Generator().manual_seed(3)
    ones = [x.to(DEV) for x in orc.init_quantized_pool(B + 1, HV, K, K, h0=torch.randn(B + 1, HV, K, K, generator=g) * 0.1,
                                                       resid_fmt=resid_fmt, resid_scale=rscale)]
    many = [x.clone() for x in ones]
    A_log, dt_bias = toks[0][3].to(DEV), toks[0][4].to(DEV)
    idx = torch.tensor([2, 0, 5, 1, 3], dtype=torch.int32, device=DEV)
    acts = [torch.stack([x[i] for x in toks], 1).to(dtype).to(DEV) for i in range(3)]
    how = dict(use_qk_l2norm_in_kernel=l2norm, resid_fmt=resid_fmt)
    for _ in range(rounds):
        outs = []
        for t in range(T):
            outs.append(torch.full((B, 1, HV, K), -3.0, dtype=out_dtype, device=DEV))
            qpd.quantized_gated_delta_rule_packed_decode(*(x[:, t].contiguous() for x in acts), A_log, dt_bias, K ** -0.5, *ones, outs[-1],
                                                         idx, **how)
            assert _lib.load_library().carry_gdn_last_kernel() == 2
        whole, out = _guarded(B, T, HV, K, out_dtype)
        qpd.quantized_gated_delta_rule_packed_decode_multi(*acts, A_log, dt_bias, K ** -0.5, *many, out, idx, **how)
        assert _lib.load_library().carry_gdn_last_kernel() == 3
        assert _same(out, torch.cat(outs, 1))
        assert bool((whole[:32] == -3.0).all()) and bool((whole[-32:] == -3.0).all())
        for x, y in zip(many, ones):
            assert _same(x, y)


@pytest.mark.parametrize("kind", ["outlier", "ladder", "zero", "tiny", "nan", "inf", "repeat"])
@pytest.mark.parametrize("resid_fmt,rscale", [(0, "v"), (0, "head"), (1, "v"), (1, "head")])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_equals_single_token_calls(kind, resid_fmt, rscale, dtype):
    B, T, H, HV, K = 5, 3, 2, 4, 128
    toks = _toks(T, B, H, HV, K, kind == "repeat")
    for t, (mixed, *_) in enumerate(toks):
        qk = mixed[:, :2 * H * K].view(B, 2 * H, K)
        if kind == "outlier":
            qk[:, :, 5] *= 2.0 ** 10
        elif kind == "ladder":
            qk *= 2.0 ** -(torch.arange(K) % 24).float()
        elif kind == "zero":
            qk[t] = 0
        elif kind == "tiny":
            qk *= 2.0 ** -20
        elif kind in ("nan", "inf") and t == 1:
            qk[2, 2 * H - 1, 9] = float(kind)                # one key of one request, in the second token
    _check(toks, H, HV, K, resid_fmt, rscale, dtype, dtype, True, rounds=32 if kind == "repeat" else 1)


@pytest.mark.parametrize("dtype,out_dtype", [(torch.float32, torch.bfloat16), (torch.float32, torch.float16),
                                             (torch.bfloat16, torch.float32), (torch.bfloat16, torch.float16),
                                             (torch.float16, torch.float32), (torch.float16, torch.float16)])
@pytest.mark.parametrize("resid_fmt,rscale", [(0, "v"), (0, "head"), (1, "v"), (1, "head")])
@pytest.mark.parametrize("l2norm", [False, True])
def test_norm_off_and_outputs_of_another_type(l2norm, resid_fmt, rscale, dtype, out_dtype):
    """q and k as they come (k_mul = 1, q_mul = the scale), and a store whose width is the output's, not the activations'."""
    B, T, H, HV, K = 5, 9, 2, 4, 128
    _check(_toks(T, B, H, HV, K, False, gain=1.0 if l2norm else K ** -0.5), H, HV, K, resid_fmt, rscale, dtype, out_dtype, l2norm)
