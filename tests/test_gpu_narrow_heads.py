"""The slot-indexed kernel for 64-wide heads against the generic kernel, which takes the same call when a slot's rows
are not on a 16-byte grid: every operation is rounded alike, so everything they leave must be equal bit for bit."""

from __future__ import annotations

import pytest
import torch

from oracle import gdn_oracle as orc
from parity import make_packed_inputs

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("B,H,HV", [(1, 1, 1), (5, 3, 6), (40, 8, 16)])
@pytest.mark.parametrize("resid_fmt,rscale", [(0, "v"), (0, "head"), (1, "v"), (1, "head")])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("l2norm", [True, False])
def test_equals_the_generic_kernel(B, H, HV, resid_fmt, rscale, dtype, l2norm):
    from carrykernel_b200 import _lib
    from carrykernel_b200.vllm_integration import quantized_packed_decode as qpd
    K = V = 64
    slots = B + 3
    g = torch.Generator().manual_seed(B)
    h0 = torch.randn(slots, HV, V, K, generator=g) * 0.1
    ref = orc.init_quantized_pool(slots, HV, V, K, h0=h0, resid_fmt=resid_fmt, resid_scale=rscale)
    dense = [t.to(DEV) for t in ref]
    odd = []                                            # the same pool with 8 more bytes between slots
    for t in dense:
        pad = 8 if t.dtype == torch.int8 else 0
        row = t[0].numel() + pad
        wide = torch.zeros(slots * row, dtype=t.dtype, device=DEV)
        view = wide.as_strided(t.shape, (row, *t.stride()[1:]))
        view.copy_(t)
        odd.append(view)
    idx = torch.randperm(slots - 1, generator=g)[:B] + 1
    if B > 1:
        idx[1], idx[2] = 0, slots                       # a padding request and a slot id beyond the pool
    idx = idx.to(torch.int32).to(DEV)
    for t in range(3):
        args = [x.to(DEV) for x in make_packed_inputs(B, H, HV, K, V, seed=t, dtype=dtype, qk_gain=1.0 if l2norm else K ** -0.5)]
        outs, kernels, bits = [], [], []
        for pool in (dense, odd):
            out = torch.full((B, 1, HV, V), float("nan"), dtype=dtype, device=DEV)
            status = torch.zeros(1, dtype=torch.int32, device=DEV)
            qpd.quantized_gated_delta_rule_packed_decode(*args, K ** -0.5, *pool, out, idx, use_qk_l2norm_in_kernel=l2norm,
                                                         resid_fmt=resid_fmt, status=status)
            outs.append(out), kernels.append(_lib.load_library().carry_gdn_last_kernel()), bits.append(int(status))
        assert kernels == [6, 1] and bits[0] == bits[1] == (_lib.STATUS_BAD_SLOT if B > 1 else 0)
        assert torch.equal(outs[0], outs[1])
        for x, y in zip(dense, odd):
            assert torch.equal(x, y)


def _same(x, y):
    """Equal, and a NaN where there is a NaN"""
    x, y = x.float(), y.float()
    return torch.equal(torch.isnan(x), torch.isnan(y)) and torch.equal(torch.nan_to_num(x, 7.0), torch.nan_to_num(y, 7.0))


@pytest.mark.parametrize("resid_fmt,rscale", [(0, "v"), (0, "head"), (1, "v"), (1, "head")])
@pytest.mark.parametrize("what", ["v nan", "v inf", "k inf", "gate nan", "scale nan", "scale inf", "resid scale nan", "resid scale inf"])
def test_equals_the_generic_kernel_on_values_that_are_not_finite(resid_fmt, rscale, what):
    """Two steps on, NaNs and infinities leave bit for bit the codes and scales that they leave in the generic kernel."""
    from carrykernel_b200 import _lib
    from carrykernel_b200.vllm_integration import quantized_packed_decode as qpd
    B, H, HV, K, V, slots = 3, 2, 4, 64, 64, 6
    g = torch.Generator().manual_seed(3)
    h0 = torch.randn(slots, HV, V, K, generator=g) * 0.1
    ref = orc.init_quantized_pool(slots, HV, V, K, h0=h0, resid_fmt=resid_fmt, resid_scale=rscale)
    mixed, a, b, A_log, dt_bias = make_packed_inputs(B, H, HV, K, V, seed=1)
    idx = torch.tensor([4, 1, 3], dtype=torch.int32, device=DEV)
    name, value = what.rsplit(" ", 1)
    hit = {"v": mixed[1, 2 * H * K + V:], "k": mixed[1, H * K:], "gate": a[1, 1:], "scale": ref[1][1, 1],
           "resid scale": ref[3].view(slots, HV, -1)[1, 1]}[name]
    hit[0] = float(value)
    acts = [x.to(DEV) for x in (mixed, a, b, A_log, dt_bias)]
    left = []
    for pad in (0, 8):                                   # 8 more bytes between slots: the generic kernel
        pool = []
        for t in ref:
            row = t[0].numel() + (pad if t.dtype == torch.int8 else 0)
            pool.append(torch.zeros(slots * row, dtype=t.dtype, device=DEV).as_strided(t.shape, (row, *t.stride()[1:])))
            pool[-1].copy_(t)
        outs = []
        for _ in range(2):
            outs.append(torch.zeros(B, 1, HV, V, device=DEV))
            qpd.quantized_gated_delta_rule_packed_decode(*acts, K ** -0.5, *pool, outs[-1], idx, use_qk_l2norm_in_kernel=True,
                                                         resid_fmt=resid_fmt)
            assert _lib.load_library().carry_gdn_last_kernel() == (1 if pad else 6)
        left.append((*outs, *pool))
    assert not torch.isfinite(left[1][0]).all() or name == "resid scale"
    for x, y in zip(*left):
        assert _same(x, y)
