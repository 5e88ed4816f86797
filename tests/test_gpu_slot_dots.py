"""Streaming kernel of the slot layout: tile counts per CTA at which its set-up or its ring changes, and activations at
which its fixed-point dot products do."""

from __future__ import annotations

import pytest
import torch

import parity
from oracle import gdn_oracle as orc
from parity import make_packed_inputs

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _call(mixed, a, b, A_log, dt_bias, pool, out, idx, resid_fmt, l2norm=True):
    from carrykernel_b200.vllm_integration import quantized_packed_decode as qpd
    qpd.quantized_gated_delta_rule_packed_decode(mixed, a, b, A_log, dt_bias, 128 ** -0.5, *pool, out, idx,
                                                 use_qk_l2norm_in_kernel=l2norm, resid_fmt=resid_fmt)


# tiles per CTA: 1, 8 and 9 (lanes per tile in the set-up), 32 and 33 (the same), up to 65 (facts beyond the cached ones)
@pytest.mark.parametrize("per_cta", [1, 2, 3, 4, 5, 8, 9, 32, 33, 48, 49, 64, 65])
@pytest.mark.parametrize("resid_fmt,rscale,dtype", [(1, "head", torch.bfloat16), (0, "v", torch.float32)])
def test_a_batch_is_its_requests(per_cta, resid_fmt, rscale, dtype):
    """Bit for bit what calls on 37 requests (at most one tile per CTA) leave, padding in between."""
    HV, H, T = 8, 4, 128
    ctas = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    B = per_cta * ctas // HV
    g = torch.Generator(device=DEV).manual_seed(per_cta)
    codes = torch.randint(-127, 128, (B + 1, HV, T, T), dtype=torch.int8, device=DEV, generator=g)
    resid = torch.randint(-127, 128, (B + 1, HV, T, T // 2 if resid_fmt == 1 else T), dtype=torch.int8, device=DEV, generator=g)
    sscale = torch.rand(B + 1, HV, T, device=DEV, generator=g) * 1e-3 + 1e-4
    rs = torch.rand(*((B + 1, HV) if rscale == "head" else (B + 1, HV, T)), device=DEV, generator=g) * 1e-5 + 1e-6
    pool = [codes, sscale, resid, rs]
    idx = (torch.randperm(B, device=DEV, generator=g) + 1).to(torch.int32)
    idx[::11] = 0
    mixed = torch.randn(B, (2 * H + HV) * T, device=DEV, generator=g).to(dtype)
    a, b = (torch.randn(B, HV, device=DEV, generator=g).to(dtype) for _ in range(2))
    A_log, dt_bias = torch.randn(HV, device=DEV, generator=g) * 0.2, torch.randn(HV, device=DEV, generator=g) * 0.1
    whole, parts = [x.clone() for x in pool], [x.clone() for x in pool]
    out_whole, out_parts = (torch.full((B, 1, HV, T), float("nan"), dtype=dtype, device=DEV) for _ in range(2))
    _call(mixed, a, b, A_log, dt_bias, whole, out_whole, idx, resid_fmt)
    for r in range(0, B, 37):
        s = slice(r, r + 37)
        _call(mixed[s], a[s], b[s], A_log, dt_bias, parts, out_parts[s], idx[s], resid_fmt)
    assert torch.equal(out_whole, out_parts) and not torch.isnan(out_whole).any()
    for x, y in zip(whole, parts):
        assert torch.equal(x, y)


def _spread(kind, x, H, K):
    """q and k of `x` [B, (2H + HV) K] made extreme; v stays."""
    qk = x[:, :2 * H * K].view(x.shape[0], 2 * H, K)
    if kind == "outlier":
        qk[:, :, 5] *= 2.0 ** 12
    elif kind == "ladder":                       # 2^0 .. 2^-31 along the vector
        qk *= 2.0 ** -(torch.arange(K) % 32).float()
    elif kind == "zero":
        qk[0] = 0; qk[1, :H] = 0; qk[2, H:] = 0
    elif kind == "tiny":                         # below what the fixed point takes
        qk *= 2.0 ** -110
    return x


@pytest.mark.parametrize("kind", ["outlier", "ladder", "zero", "tiny"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("l2norm", [True, False])
def test_activations_of_extreme_sizes(kind, dtype, l2norm):
    B, H, HV, K = 4, 2, 4, 128
    g = torch.Generator().manual_seed(2)
    ref = list(orc.init_quantized_pool(B + 1, HV, K, K, h0=torch.randn(B + 1, HV, K, K, generator=g) * 0.1,
                                       resid_fmt=orc.RESID_INT4, resid_scale="v"))
    mixed, a, b, A_log, dt_bias = make_packed_inputs(B, H, HV, K, K, seed=3, qk_gain=K ** -0.5)
    mixed = _spread(kind, mixed, H, K).to(dtype)
    idx = torch.tensor([2, 4, 1, 3], dtype=torch.int32)
    got = [x.clone().to(DEV) for x in ref]
    out = torch.full((B, 1, HV, K), float("nan"), device=DEV)
    _call(mixed.to(DEV), a.to(DEV).to(dtype), b.to(DEV).to(dtype), A_log.to(DEV), dt_bias.to(DEV), got, out, idx.to(DEV), 1, l2norm)
    want = torch.empty(B, 1, HV, K)
    orc.packed_decode_step(mixed, a.to(dtype), b.to(dtype), A_log, dt_bias, K ** -0.5, *ref, want, idx, use_qk_l2norm_in_kernel=l2norm,
                           resid_fmt=orc.RESID_INT4)
    # per head: an output is a sum of 128 products, 2e-5 of the largest covers its roundings in fp32
    off = (out.cpu() - want).abs().amax(-1) / want.abs().amax(-1).clamp(min=1e-37)
    assert float(off.max()) < 2e-5
    # not with a raw k of 362: <h, k> is then 36 or so against v of about 1, some of the 2048 rows have a dv (and so a scale)
    # that is a hundredth of what it is the difference of, and 1.2e-7 of that is more than the 1e-5 that scales may be off
    if l2norm or kind != "outlier":
        parity.check_pool(got, ref, True, idx.tolist(), orc.unpack_int4, f"{kind} {dtype}")


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("where", ["q", "k"])
def test_not_finite_stays_with_its_request(value, where):
    """One request's q or k has an element that is not finite: its outputs are what the generic kernel's are (found NaN in the
    same places), every other request's are untouched by it."""
    B, H, HV, K = 5, 4, 4, 128
    g = torch.Generator().manual_seed(4)
    st = [x.to(DEV) for x in orc.init_quantized_pool(B + 1, HV, K, K, h0=torch.randn(B + 1, HV, K, K, generator=g) * 0.1,
                                                     resid_fmt=orc.RESID_INT8, resid_scale="v")]
    mixed, a, b, A_log, dt_bias = [x.to(DEV) for x in make_packed_inputs(B, H, HV, K, K, seed=5)]
    idx = torch.arange(1, B + 1, dtype=torch.int32, device=DEV)
    bad = mixed.clone()
    bad[2, (0 if where == "q" else H * K) + K + 7] = value            # request 2, key head 1
    outs, pools = [], []
    wide = torch.zeros(B, mixed.shape[1] + 1, device=DEV)             # rows off the 16-byte grid: the generic kernel
    wide[:, :-1] = bad
    for x in (mixed, bad, wide[:, :-1]):
        pool, out = [y.clone() for y in st], torch.zeros(B, 1, HV, K, device=DEV)
        _call(x, a, b, A_log, dt_bias, pool, out, idx, 0)
        outs.append(out); pools.append(pool)
    keep = torch.ones(B, HV, dtype=torch.bool, device=DEV)
    keep[2, 1] = False
    assert torch.equal(outs[1][:, 0][keep], outs[0][:, 0][keep])
    for x, y in zip(pools[1], pools[0]):
        assert torch.equal(x[1:][keep], y[1:][keep])
    assert torch.equal(torch.isnan(outs[1][2, 0, 1]), torch.isnan(outs[2][2, 0, 1])) and torch.isnan(outs[1][2, 0, 1]).any()
