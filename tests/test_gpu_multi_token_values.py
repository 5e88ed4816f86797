"""Multi-token call against single-token calls, bit for bit, on activations that are zero, far apart in size, not finite or the
same for 96 tokens (codes settle at rounding ties then, and most tiles have some to decide again): the two kernels split a tile
differently, and must still take every sum and maximum alike."""

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


@pytest.mark.parametrize("kind", ["outlier", "ladder", "zero", "tiny", "nan", "inf", "repeat"])
@pytest.mark.parametrize("resid_fmt,rscale", [(0, "v"), (0, "head"), (1, "v"), (1, "head")])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_equals_single_token_calls(kind, resid_fmt, rscale, dtype):
    from carrykernel_b200 import _lib
    from carrykernel_b200.vllm_integration import quantized_packed_decode as qpd
    B, T, H, HV, K = 5, 3, 2, 4, 128
    g = torch.Generator().manual_seed(3)
    ref = [x.to(DEV) for x in orc.init_quantized_pool(B + 1, HV, K, K, h0=torch.randn(B + 1, HV, K, K, generator=g) * 0.1,
                                                      resid_fmt=resid_fmt, resid_scale=rscale)]
    toks = [list(make_packed_inputs(B, H, HV, K, K, seed=7 if kind == "repeat" else 7 + t)) for t in range(T)]
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
    A_log, dt_bias = toks[0][3].to(DEV), toks[0][4].to(DEV)
    idx = torch.tensor([2, 0, 5, 1, 3], dtype=torch.int32, device=DEV)
    acts = [torch.stack([x[i] for x in toks], 1).to(dtype).to(DEV) for i in range(3)]
    ones, many = [x.clone() for x in ref], [x.clone() for x in ref]
    for _ in range(32 if kind == "repeat" else 1):
        outs = []
        for t in range(T):
            outs.append(torch.full((B, 1, HV, K), -3.0, dtype=dtype, device=DEV))
            qpd.quantized_gated_delta_rule_packed_decode(*(x[:, t].contiguous() for x in acts), A_log, dt_bias, K ** -0.5, *ones, outs[-1],
                                                         idx, use_qk_l2norm_in_kernel=True, resid_fmt=resid_fmt)
            assert _lib.load_library().carry_gdn_last_kernel() == 2
        out = torch.full((B, T, HV, K), -3.0, dtype=dtype, device=DEV)
        qpd.quantized_gated_delta_rule_packed_decode_multi(*acts, A_log, dt_bias, K ** -0.5, *many, out, idx, use_qk_l2norm_in_kernel=True,
                                                           resid_fmt=resid_fmt)
        assert _lib.load_library().carry_gdn_last_kernel() == 3
        assert _same(out, torch.cat(outs, 1))
        for x, y in zip(many, ones):
            assert _same(x, y)
