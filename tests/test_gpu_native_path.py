"""Every surface with and without the native call path: the checks in Python and ctypes launch the same kernels."""

from __future__ import annotations

import pytest
import torch

from parity import make_packed_inputs, seeded_inputs

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _everything():
    from carrykernel_b200.statequant import kernel as sq
    from carrykernel_b200.vllm_integration import quantized_packed_decode as qpd
    from carrykernel_b200.vllm_integration import state_pool as sp
    from carrykernel_b200.vllm_integration.state_cache import SlotCache
    left = []
    for edge, fmt in ((128, sq.RES_INT8), (64, sq.RES_INT4), (16, sq.RES_FP16), (128, sq.RES_NONE)):
        h0, q, k, v, alpha, beta = [x.to(DEV) for x in seeded_inputs(2, 4, edge, edge, seed=edge, alpha_mode="gated")]
        left += sq.gdn_quant_step_fused(*sq.init_quant_state(h0, 8, fmt), q, k, v, alpha, beta, res_fmt=fmt)
        left += sq.gdn_step_fused_fp32(h0, q, k, v, alpha, beta)
        h0, *acts = [x.to(DEV) for x in seeded_inputs(2, 4, edge, edge, seed=edge, T=3, alpha_mode="gated")]
        for res in (fmt, sq.RES_FP32):
            left += sq.gdn_quant_decode_fused(h0, *acts, 3, res_fmt=res)
    for edge in (128, 64):
        c = SlotCache(2, 5, 4, edge, edge, DEV, qpd.RESID_INT4, "head", spill_slots=3)
        c.allocate("a"), c.allocate("b")
        idx = c.indices(["b", "a"], pad_to=3)
        h = (torch.randn(3, 4, edge, edge, generator=torch.Generator().manual_seed(edge)) * 0.1).to(DEV)
        mixed, a, b, A_log, dt_bias = [x.to(DEV) for x in make_packed_inputs(3, 2, 4, edge, edge, seed=edge)]
        for pool in c.pools:
            sp.store_state(h, pool, idx, resid_fmt=qpd.RESID_INT4, keep_error=True)
            out = torch.zeros(3, 1, 4, edge, device=DEV)
            qpd.quantized_gated_delta_rule_packed_decode(mixed, a, b, A_log, dt_bias, 0.1, *pool, out, idx, resid_fmt=qpd.RESID_INT4)
            outs = torch.zeros(3, 2, 4, edge, device=DEV)
            two = [torch.stack([x, x], 1).contiguous() for x in (mixed, a, b)]
            qpd.quantized_gated_delta_rule_packed_decode_multi(*two, A_log, dt_bias, 0.1, *pool, outs, idx, resid_fmt=qpd.RESID_INT4)
            sp.copy_slots(pool, idx[:1].contiguous(), torch.tensor([4], dtype=torch.int32, device=DEV), resid_fmt=qpd.RESID_INT4)
            left += [out, outs, sp.load_state(pool, idx, resid_fmt=qpd.RESID_INT4, out=torch.zeros_like(h))]
        c.preempt("a")
        c.fork("b", "c")
        c.resume("a")
        left += [t for pool in c.pools for t in pool] + [idx, c.indices(["a", "b", "c"])]
    torch.cuda.synchronize()
    return [None if t is None else t.cpu() for t in left]


def test_without_the_native_call_path(monkeypatch):
    from carrykernel_b200 import _lib
    lib = _lib.load_library()
    with_it = _everything()
    monkeypatch.setattr(lib, "native", _lib._NoNative())
    without = _everything()
    assert len(with_it) == len(without)
    for x, y in zip(with_it, without):
        assert (x is None) == (y is None) and (x is None or torch.equal(x.float(), y.float()))
