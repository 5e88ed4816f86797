"""Multi-token call of the slot-indexed path: T tokens per request in one launch.

The contract is "T single-token calls, bit for bit", so the main check is
exact equality with the single-token kernel (itself parity-tested against the
oracle); one case is also compared with the CPU oracle directly."""

from __future__ import annotations

import pytest
import torch

import parity
from oracle import gdn_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _qpd():
    from carrykernel_b200.vllm_integration import quantized_packed_decode as qpd
    return qpd


def _inputs(B, T, H, HV, K, V, seed, dtype):
    g = torch.Generator().manual_seed(seed)
    q = torch.randn(B, T, H * K, generator=g)
    k = torch.randn(B, T, H * K, generator=g)
    v = torch.randn(B, T, HV * V, generator=g)
    mixed = torch.cat([q, k, v], dim=2).contiguous().to(dtype)
    a = (torch.randn(B, T, HV, generator=g) * 0.5).to(dtype)
    b = torch.randn(B, T, HV, generator=g).to(dtype)
    A_log = torch.randn(HV, generator=g) * 0.2
    dt_bias = torch.randn(HV, generator=g) * 0.1
    return mixed, a, b, A_log, dt_bias


def _pool(num_slots, HV, V, K, resid_fmt, rscale, seed):
    g = torch.Generator().manual_seed(seed)
    pool = torch.randn(num_slots, HV, V, K, generator=g) * 0.1
    return list(orc.init_quantized_pool(num_slots, HV, V, K, h0=pool, resid_fmt=resid_fmt, resid_scale=rscale))


def _check_equals_single_token_calls(T, resid_fmt, rscale, dtype, H=16, HV=32):
    qpd = _qpd()
    from carrykernel_b200 import _lib
    B, K, V = 5, 128, 128
    num_slots = 9
    st = _pool(num_slots, HV, V, K, resid_fmt, rscale, seed=11)
    mixed, a, b, A_log, dt_bias = _inputs(B, T, H, HV, K, V, 5, dtype)
    idx = torch.tensor([3, 0, 8, 1, 5], dtype=torch.int32)        # one padding request
    dev = lambda x: x.to(DEV)
    # T single-token calls
    ref = [dev(x.clone()) for x in st]
    out_ref = torch.full((B, T, HV, V), float("nan"), dtype=dtype, device=DEV)
    for t in range(T):
        tmp = torch.empty(B, 1, HV, V, dtype=dtype, device=DEV)
        qpd.quantized_gated_delta_rule_packed_decode(
            dev(mixed[:, t].contiguous()), dev(a[:, t].contiguous()), dev(b[:, t].contiguous()), dev(A_log),
            dev(dt_bias), K ** -0.5, *ref, tmp, dev(idx), use_qk_l2norm_in_kernel=True, resid_fmt=resid_fmt)
        out_ref[:, t:t + 1] = tmp
    # one multi-token call
    got = [dev(x.clone()) for x in st]
    out = torch.full((B, T, HV, V), float("nan"), dtype=dtype, device=DEV)
    qpd.quantized_gated_delta_rule_packed_decode_multi(
        dev(mixed), dev(a), dev(b), dev(A_log), dev(dt_bias), K ** -0.5, *got, out, dev(idx),
        use_qk_l2norm_in_kernel=True, resid_fmt=resid_fmt)
    torch.cuda.synchronize()
    assert _lib.load_library().carry_gdn_last_kernel() == 3, "the multi-token kernel should have served this shape"
    assert torch.equal(out, out_ref)
    for x, y in zip(got, ref):
        assert torch.equal(x, y)
    assert torch.all(out[1] == 0)


@pytest.mark.parametrize("resid_fmt", [orc.RESID_INT4, orc.RESID_INT8])
@pytest.mark.parametrize("rscale", ["head", "v"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_multi_equals_single_token_calls(resid_fmt, rscale, dtype):
    _check_equals_single_token_calls(3, resid_fmt, rscale, dtype)


@pytest.mark.parametrize("T", [1, 7, 8, 9, 17])
@pytest.mark.parametrize("resid_fmt", [orc.RESID_INT4, orc.RESID_INT8])
@pytest.mark.parametrize("rscale", ["head", "v"])
def test_multi_equals_single_token_calls_across_chunks_of_activations(T, resid_fmt, rscale):
    """The kernel fetches the activations of 8 tokens at a time; the refill is the only block barrier between tokens."""
    _check_equals_single_token_calls(T, resid_fmt, rscale, torch.float16, H=4, HV=8)


def test_multi_against_oracle():
    qpd = _qpd()
    B, T, H, HV, K, V = 3, 2, 8, 16, 128, 128
    num_slots = 5
    st = _pool(num_slots, HV, V, K, orc.RESID_INT4, "head", seed=2)
    mixed, a, b, A_log, dt_bias = _inputs(B, T, H, HV, K, V, 9, torch.bfloat16)
    idx = torch.tensor([4, 2, 1], dtype=torch.int32)
    ref = [x.clone() for x in st]
    out_ref = torch.empty(B, T, HV, V, dtype=torch.bfloat16)
    orc.packed_decode_multi(mixed, a, b, A_log, dt_bias, K ** -0.5, *ref, out_ref, idx,
                            use_qk_l2norm_in_kernel=True, resid_fmt=orc.RESID_INT4)
    got = [x.clone().to(DEV) for x in st]
    out = torch.empty(B, T, HV, V, dtype=torch.bfloat16, device=DEV)
    qpd.quantized_gated_delta_rule_packed_decode_multi(
        mixed.to(DEV), a.to(DEV), b.to(DEV), A_log.to(DEV), dt_bias.to(DEV), K ** -0.5, *got, out, idx.to(DEV),
        use_qk_l2norm_in_kernel=True, resid_fmt=qpd.RESID_INT4)
    torch.cuda.synchronize()
    parity.assert_close(out.cpu(), out_ref, "multi: out", rtol=8e-3, atol=1e-4)
    # free-running over two tokens: an ulp of difference after the first token is an input of the second
    # (and a residual scale that moved by 1e-4 re-rounds a visible fraction of the next token's codes), so
    # codes are not compared one by one here -- that is what the bit-exact test above is for; scales are
    # compared at 1e-4 instead of the teacher-forced 1e-5, and what the codes stand for, state plus
    # carried residual, as below
    live = idx.long()
    sc, ss, rc, rs = [x.cpu() for x in got]
    torch.testing.assert_close(ss[live], ref[1][live], rtol=1e-4, atol=1e-30)
    torch.testing.assert_close(rs[live], ref[3][live], rtol=5e-3, atol=1e-30)
    h_got = sc[live].float() * ss[live][..., None] + orc.unpack_int4(rc[live]).float() * rs[live][..., None, None]
    h_ref = ref[0][live].float() * ref[1][live][..., None] + orc.unpack_int4(ref[2][live]).float() * ref[3][live][..., None, None]
    # within one state step everywhere (the bound the single-step protocol uses at flipped elements), and
    # within a residual step nearly everywhere
    err = (h_got - h_ref).abs()
    assert float(err.max()) <= float(ref[1][live].max())
    assert float((err > ref[3][live][..., None, None]).float().mean()) <= 1e-3


def test_multi_falls_back_for_other_shapes():
    qpd = _qpd()
    B, T, H, HV, K, V = 3, 2, 2, 4, 64, 32
    st = _pool(5, HV, V, K, orc.RESID_INT8, "v", seed=4)
    mixed, a, b, A_log, dt_bias = _inputs(B, T, H, HV, K, V, 3, torch.float32)
    idx = torch.tensor([1, 4, 2], dtype=torch.int32)
    dev = lambda x: x.to(DEV)
    ref = [dev(x.clone()) for x in st]
    out_ref = torch.empty(B, T, HV, V, device=DEV)
    for t in range(T):
        tmp = torch.empty(B, 1, HV, V, device=DEV)
        qpd.quantized_gated_delta_rule_packed_decode(
            dev(mixed[:, t].contiguous()), dev(a[:, t].contiguous()), dev(b[:, t].contiguous()), dev(A_log),
            dev(dt_bias), K ** -0.5, *ref, tmp, dev(idx), use_qk_l2norm_in_kernel=True, resid_fmt=orc.RESID_INT8)
        out_ref[:, t:t + 1] = tmp
    got = [dev(x.clone()) for x in st]
    out = torch.empty(B, T, HV, V, device=DEV)
    qpd.quantized_gated_delta_rule_packed_decode_multi(
        dev(mixed), dev(a), dev(b), dev(A_log), dev(dt_bias), K ** -0.5, *got, out, dev(idx),
        use_qk_l2norm_in_kernel=True, resid_fmt=orc.RESID_INT8)
    torch.cuda.synchronize()
    assert torch.equal(out, out_ref)
    for x, y in zip(got, ref):
        assert torch.equal(x, y)
